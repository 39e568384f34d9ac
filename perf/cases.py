"""What this framework is timed on: the passes that its users' programs make.

A case is a dict of plain values.  ``kind`` says which program it stands for:

* ``flow``: a simulation through ``Solver`` (the reference programs' main
  loop): some steps, then the populations read into a page-locked buffer, and
  the running statistics where the record collects them.
* ``calls``: the kernel-level functions on a caller's own device buffers: one
  stream-collide step and the body force of the same populations.
* ``boxes``: the ensemble of periodic boxes: data generation for the closure
  (seeded turbulence, steps, energies, filtered samples), or boxes run with a
  subgrid model from given populations (steps, velocities).
* ``fit``: training of the closure on device samples.
* ``evaluate``: validation of a closure: loss and gradient over all samples,
  and the predictions of both inference paths.

``exact`` restates each in 64-bit torch from the documented equations.
"""
import ctypes
import functools
import math

import numpy as np
import torch

import lbm_multigpu_gb300 as lbm

DEV = "cuda"
BYTES = {"fp32": 4, "fp16": 2, "bf16": 2, "fp64": 8}
FLOP_NODE = 270          # one MRT + Smagorinsky node update
FLOP_MLP = 10_240        # 2 (16 * 64 + 64 * 64 + 64), the closure's forward pass
P_REF, NU_SCALE = 0.01, 1e-4
TMAX = 1_000_000         # the length of the run that a pass is a part of


def listed():
    flow = dict(kind="flow", geometry="channel_square", model="MRT", les=True, halfway=True, noise=True, stats=False,
                precision="fp32", closure_every=0, tau=0.52, refined=False)
    return [
        # a host program with its own buffers and step loop (FFI, coupling): latency
        dict(name="calls_96", kind="calls", nx=96, ny=48, nz=33, pitch=96, model="MRT", les=True, tau=0.55),
        # the lid-driven cavity configuration: a small domain, many steps
        dict(flow, name="cavity_64", geometry="cavity", model="BGK", les=False, halfway=False, noise=False, tau=0.6,
             nx=64, ny=64, nz=64, steps=250),
        # a parameter-study channel of ragged sizes, the reference's full-way walls, running statistics
        dict(flow, name="channel_ragged", halfway=False, noise=False, stats=True, nx=211, ny=70, nz=45, steps=400),
        # the channel that the throughput metric is quoted on
        dict(flow, name="channel_512", nx=512, ny=128, nz=128, steps=100),
        # the same with half the memory per node (long runs on large domains)
        dict(flow, name="channel_512_fp16", precision="fp16", nx=512, ny=128, nz=128, steps=100),
        # the 64-bit twin that precision studies compare with
        dict(flow, name="channel_fp64", precision="fp64", nx=256, ny=64, nz=64, steps=40),
        # the learned closure deployed in the channel, evaluated on every step
        dict(flow, name="channel_closure", closure_every=1, nx=512, ny=128, nz=128, steps=40),
        # the two-level refinement configuration: cylinder in a fine patch, linear time interpolation
        dict(flow, name="refined", geometry="channel_circle", halfway=False, refined=True, nx=256, ny=128, nz=64,
             steps=100),
        # data generation for the closure: boxes of uneven sizes from seeded turbulence
        dict(name="boxes_generate", kind="boxes", sizes="64,112,80,128,96,48,112,72", sgs="none", steps=200),
        # the a-posteriori test of the closure: coarse boxes with the network
        dict(name="boxes_closure", kind="boxes", sizes="64,80,32,56,48,72,40,64", sgs="mlp", steps=50),
        # training of the closure at the pipeline's batch size
        dict(name="fit", kind="fit", n=262_144, batch=16_384, steps=32),
        # validation of a trained closure on held-out samples
        dict(name="evaluate", kind="evaluate", n=1_000_003),
    ]


def _spread(rng, lo, hi):
    """a whole number from lo to hi, even in its logarithm"""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["flow"] * 5 + ["calls", "refined", "boxes", "boxes", "fit", "evaluate"])
    if kind == "calls":
        nx = _spread(rng, 20, 400)
        return dict(kind="calls", nx=nx, ny=_spread(rng, 12, 120), nz=_spread(rng, 5, 80),
                    pitch=(nx + 31) // 32 * 32 + rng.choice([0, 0, 32]), model=rng.choice(["MRT", "MRT", "MRT_DI3", "BGK"]),
                    les=rng.random() < 0.7, tau=rng.choice([0.53, 0.55, 0.6]))
    if kind == "refined":
        return dict(kind="flow", geometry="channel_circle", model="MRT", les=True, halfway=False, noise=rng.random() < 0.5,
                    stats=False, precision=rng.choice(["fp32", "fp32", "fp16"]), closure_every=0, tau=0.52, refined=True,
                    nx=_spread(rng, 100, 300), ny=_spread(rng, 64, 140), nz=_spread(rng, 32, 80), steps=_spread(rng, 10, 80))
    if kind == "flow":
        closed = rng.random() < 0.2
        nodes = _spread(rng, 10_000, 8_000_000)
        side = nodes ** (1 / 3)
        a, b = rng.uniform(0.6, 1.1), rng.uniform(0.6, 1.1)
        ny, nz = max(14, round(side * a)), max(6, round(side * b))
        nx = max(24, round(nodes / (ny * nz)))
        precision = rng.choice(["fp32", "fp32", "fp32", "fp16", "fp16", "bf16", "fp64"])
        if precision == "fp64":
            nx = max(24, min(nx, 1_000_000 // (ny * nz)))
        model = rng.choice(["MRT", "MRT", "MRT", "BGK", "MRT_DI3"])
        closure = 0
        if not closed and model == "MRT" and precision != "fp64" and rng.random() < 0.3:
            closure = rng.choice([1, 4, 16])
        most = 4.0e8 if closure == 1 else 2.0e7 if precision == "fp64" else 8.0e8
        steps = max(10, min(_spread(rng, 20, 400), int(most / (nx * ny * nz))))
        return dict(kind="flow", geometry="cavity" if closed else rng.choice(["channel_square", "channel_circle"]),
                    model=model, les=not closed or rng.random() < 0.5, halfway=rng.random() < 0.6,
                    noise=not closed and rng.random() < 0.6, stats=rng.random() < 0.2, precision=precision,
                    closure_every=closure, tau=rng.choice([0.52, 0.55, 0.6]), refined=False, nx=nx, ny=ny, nz=nz,
                    steps=steps)
    if kind == "boxes":
        sgs = rng.choice(["none", "none", "smagorinsky", "mlp"])
        top = 128 if sgs == "none" else 80
        sizes = [2 * _spread(rng, 8, top // 2) for _ in range(rng.randint(1, 8))]
        return dict(kind="boxes", sizes=",".join(map(str, sizes)), sgs=sgs, steps=_spread(rng, 8, 150))
    if kind == "fit":
        n = _spread(rng, 4_000, 400_000)
        return dict(kind="fit", n=n, batch=min(n, _spread(rng, 500, 32_768)), steps=_spread(rng, 8, 40))
    return dict(kind="evaluate", n=_spread(rng, 1_000, 1_000_000))


# ---------------------------------------------------------------- the records

def _body(case):
    """centre and half side (radius) of the body"""
    nx, ny = case["nx"], case["ny"]
    return nx // 4 + 0.5, ny // 2 - 0.5, float(max(2, ny // 16))


def _patch(case):
    """the refinement patch: fine sizes and origin (ratio 2, bounded in z, around the body)"""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    cx, cy, r = _body(case)
    px, py, pz = max(3 * nx // 8, int(12 * r)) // 4 * 4, ny // 2 // 4 * 4, nz // 4 * 4
    return (px, py, pz), (max(1, int(cx - 2 * r)) + 0.25, int(cy - py / 4) + 0.25, nz // 4 + 0.25)


def _record(case, seed):
    cx, cy, r = _body(case)
    ext = {}
    if case["refined"]:
        dims, origin = _patch(case)
        ext.update(refinement=1, lr_dims=dims, lr_factor=0.5, lr_origin=origin, cf_time="linear")
    if case["closure_every"]:
        ext.update(sgs="mlp", sgs_every=case["closure_every"])
    if case["geometry"] == "cavity":
        ext.update(lid_velocity=(0.05, 0.0, 0.0), lid_face="+z")
    if case["noise"]:
        ext.update(inlet_noise=0.01, seed=seed % 1_000_003)
    if case["stats"]:
        ext.update(velav=1, start_velav=0, start_velfluc=max(1, case["steps"] // 2))
    if case["halfway"]:
        ext.update(bounceback="halfway")
    return lbm.make_inputs(case["nx"], case["ny"], case["nz"], obst1=(cx, cy, 0.0), r1=r, re=120.0, umax=0.05,
                           tmax=TMAX, les=int(case["les"]), cs=0.01, model=case["model"], geometry=case["geometry"],
                           precision=case["precision"], tau=case["tau"], **ext)


# ---------------------------------------------------------------- inputs

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _waves(shape, amp, gen):
    """a smooth periodic velocity field [3][nz][ny][nx] of rms about amp (64 bits)"""
    nz, ny, nx = shape
    u = torch.zeros((3, nz, ny, nx), dtype=torch.float64, device=DEV)
    r = torch.rand((3, 4, 4), generator=gen, device=DEV, dtype=torch.float64).cpu()
    ax = [torch.arange(n, device=DEV, dtype=torch.float64) * (2 * math.pi / n) for n in (nz, ny, nx)]
    for c in range(3):
        for m in range(4):
            k = [int(v * 4) + (1 if c != d else 0) for d, v in enumerate(r[c, m, :3].tolist())]
            ph = 2 * math.pi * float(r[c, m, 3])
            arg = k[0] * ax[0][:, None, None] + k[1] * ax[1][None, :, None] + k[2] * ax[2][None, None, :]
            u[c] += amp * torch.cos(arg + ph) / math.sqrt(2.0)
    return u


def _start(model, shape, base, seed):
    """populations float32[19][nz][ny][nx]: the model's equilibrium at density 1 and a disturbed velocity"""
    u = _waves(shape, 0.004, _gen(seed))
    u[0] += base
    return _equilibrium(model, torch.ones(shape, dtype=torch.float64, device=DEV), u).float()


def _samples(n, seed):
    """closure samples as filtered flows give them: |p|, the third invariant, the viscosity, and coefficients"""
    g = _gen(seed)
    X = torch.zeros((n, 16), device=DEV)
    X[:, 12] = 0.3 * torch.exp(0.8 * torch.randn(n, generator=g, device=DEV))
    X[:, 13] = (torch.rand(n, generator=g, device=DEV) * 2 - 1) * (1 / math.sqrt(6))
    X[:, 14] = torch.where(torch.rand(n, generator=g, device=DEV) < 0.5, 0.5, 2.0)
    X[:, 15] = 1.0
    T = NU_SCALE * torch.relu(0.6 + 0.8 * X[:, 13] + 0.3 * torch.randn(n, generator=g, device=DEV))
    return X, T


def _weights():
    return np.fromfile(lbm.LIB_PATH.parent.parent / "data" / "sgs_mlp.bin", np.float32)


def _fresh_params(seed):
    p = np.zeros(lbm.library().lbm_mlp_param_count(), np.float32)
    lbm._check(lbm.library().lbm_mlp_init_params(seed % 65_521, p.ctypes.data_as(ctypes.c_void_p)))
    return p


def _calls_mask(case):
    """walls y = 0 / ny - 1, inlet, outlet and a square body, in the kernel-level node types"""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    m = torch.zeros((nz, ny, case["pitch"]), dtype=torch.uint8, device=DEV)
    r = max(2, min(nx, ny) // 8)
    m[:, ny // 2 - r:ny // 2 + r, nx // 4:nx // 4 + 2 * r] = lbm.NODE["BODY"]
    m[:, :, 0] = lbm.NODE["WEST_INLET"]
    m[:, :, nx - 1] = lbm.NODE["EAST_OUTLET"]
    m[:, 0] = m[:, ny - 1] = lbm.NODE["WALL"]
    return m


def _sizes(case):
    return [int(v) for v in case["sizes"].split(",")]


def _box_start(n, m, seed):
    return _start("BGK", (n, n, n), 0.0, seed * 64 + m)


def _box_tau(case):
    return 0.51 if case["sgs"] == "none" else 0.505


def prepare(case, seed):
    kind = case["kind"]
    if kind == "calls":
        shape = (case["nz"], case["ny"], case["nx"])
        a = torch.zeros((19, case["nz"], case["ny"], case["pitch"]), device=DEV)
        a[..., :case["nx"]] = _start(case["model"], shape, 0.05, seed)
        return dict(case=case, a=a, b=torch.zeros_like(a), mask=_calls_mask(case),
                    force=torch.zeros(3, dtype=torch.float64, device=DEV),
                    scratch=torch.zeros(int(lbm.library().lbm_body_force_scratch_doubles()), dtype=torch.float64,
                                        device=DEV))
    if kind == "flow":
        s = lbm.Solver(_record(case, seed))
        if case["closure_every"]:
            s.set_sgs_mlp(_weights())
        out = []
        base = 0.0 if case["geometry"] == "cavity" else 0.05
        for level in range(s.nlevels):
            nx, ny, nz = s.dims(level)
            host = torch.empty((19, nz, ny, nx), pin_memory=True)
            host.copy_(_start(case["model"], (nz, ny, nx), base, seed + level))
            s.set_populations(host.numpy(), level)
            out.append(host.numpy())
        return dict(case=case, solver=s, out=out)
    if kind == "boxes":
        sizes = _sizes(case)
        e = lbm.Ensemble(sizes, _box_tau(case), sgs=case["sgs"], cs=0.01)
        if case["sgs"] == "none":
            e.autotune()
            cap = sum((n // 2) ** 3 for n in sizes)
            return dict(case=case, boxes=e, seed=seed % 1_000_003, cap=cap, X=torch.zeros((cap, 16), device=DEV),
                        T=torch.zeros(cap, device=DEV))
        for m, n in enumerate(sizes):
            e.set_populations(m, _box_start(n, m, seed).cpu().numpy())
        if case["sgs"] == "mlp":
            e.set_mlp(_weights())
        return dict(case=case, boxes=e)
    X, T = _samples(case["n"], seed)
    if kind == "fit":
        return dict(case=case, X=X, T=T, params=_fresh_params(seed), seed=seed % 1_000_003)
    params = _weights() + np.float32(0.02) * _fresh_params(seed)
    return dict(case=case, X=X, T=T, params=params, device_params=torch.from_numpy(params).to(DEV),
                grad=torch.zeros(params.size, device=DEV), loss=torch.zeros(1, device=DEV),
                o=torch.zeros(case["n"], device=DEV), o_tc=torch.zeros(case["n"], device=DEV))


# ---------------------------------------------------------------- one pass

def _at(t):
    return ctypes.c_void_p(t.data_ptr())


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def run(state):
    case = state["case"]
    kind = case["kind"]
    lib = lbm.library()
    if kind == "calls":
        a, b, m, force = state["a"], state["b"], state["mask"], state["force"]
        dims = (case["nx"], case["ny"], case["nz"], case["pitch"])
        force.zero_()
        lbm._check(lib.lbm_body_force_f32(_at(a), _at(m), *dims, _at(force), _at(state["scratch"]), _stream()))
        lbm._check(lib.lbm_stream_collide_f32(_at(a), _at(b), _at(m), *dims, lbm.MODELS[case["model"]],
                                              int(case["les"]), 1.0 / case["tau"], 0.01, 0.05, 1.0, 0, _stream()))
        return dict(f=b, force=force)
    if kind == "flow":
        s = state["solver"]
        s.step(case["steps"])
        got = {"f%d" % k: s.populations(k, out=o) for k, o in enumerate(state["out"])}
        if case["stats"]:
            got["stats"] = s.stats()
        return got
    if kind == "boxes":
        e = state["boxes"]
        if case["sgs"] != "none":
            e.step(case["steps"])
            return [e.velocity(m) for m in range(len(e.sizes))]
        e.init_turbulence(state["seed"])
        e.step(case["steps"])
        energy = e.energy()
        n = e.samples_into(state["X"].data_ptr(), state["T"].data_ptr(), state["cap"], 0, 0.505)
        return dict(energy=energy, X=state["X"][:n], T=state["T"][:n])
    n = case["n"]
    if kind == "fit":
        params, hist = state["params"].copy(), np.zeros(case["steps"], np.float32)
        lbm._check(lib.lbm_mlp_train(_at(state["X"]), _at(state["T"]), n, case["batch"], case["steps"], 2e-3,
                                     state["seed"], params.ctypes.data_as(ctypes.c_void_p),
                                     hist.ctypes.data_as(ctypes.c_void_p), _stream()))
        return dict(params=params, loss=hist)
    lbm._check(lib.lbm_mlp_grad(_at(state["device_params"]), _at(state["X"]), _at(state["T"]), n, _at(state["grad"]),
                                _at(state["loss"]), _stream()))
    lbm._check(lib.lbm_mlp_predict(_at(state["device_params"]), _at(state["X"]), n, _at(state["o"]), _stream()))
    lbm._check(lib.lbm_mlp_predict_tc(state["params"].ctypes.data_as(ctypes.c_void_p), _at(state["X"]), n,
                                      _at(state["o_tc"]), _stream()))
    return dict(grad=state["grad"], loss=state["loss"], o=state["o"], o_tc=state["o_tc"])


def work(case):
    kind = case["kind"]
    if kind == "calls":
        n = case["nx"] * case["ny"] * case["nz"]
        return dict(bytes=153 * n, flops=FLOP_NODE * n)
    if kind == "flow":
        n = case["nx"] * case["ny"] * case["nz"]
        nodes, steps = n, n * case["steps"]
        if case["refined"]:
            f = math.prod(_patch(case)[0])
            nodes, steps = n + f, (n + 2 * f) * case["steps"]
        per = 38 * BYTES[case["precision"]] + 1 + (16 if case["stats"] else 0) + (4 if case["closure_every"] > 1 else 0)
        every = case["closure_every"]
        return dict(bytes=per * steps + (76 + (16 if case["stats"] else 0)) * nodes,
                    flops=(FLOP_NODE + (FLOP_MLP / every if every else 0)) * steps)
    if kind == "boxes":
        n = sum(v ** 3 for v in _sizes(case))
        flops = FLOP_NODE + (FLOP_MLP if case["sgs"] == "mlp" else 0)
        if case["sgs"] != "none":
            return dict(bytes=(152 * case["steps"] + 12) * n, flops=flops * case["steps"] * n)
        # start: populations written; samples: populations read, 68 bytes per coarse cell written
        modes = sum(v ** 3 * _mode_count(v) for v in _sizes(case))
        return dict(bytes=(152 * case["steps"] + 76 + 76 + 68 / 8) * n, flops=flops * case["steps"] * n + 8 * modes)
    n = case["n"]
    if kind == "fit":
        m = case["batch"] * case["steps"]
        return dict(bytes=68 * m, flops=3 * FLOP_MLP * m)
    return dict(bytes=(3 * 64 + 4 + 8) * n, flops=5 * FLOP_MLP * n)


# ---------------------------------------------------------------- the same in 64 bits

CX = (0, 1, 0, -1, 0, 1, -1, -1, 1, 0, 1, 0, -1, 0, 0, 1, 0, -1, 0)
CY = (0, 0, 1, 0, -1, 1, 1, -1, -1, 0, 0, 1, 0, -1, 0, 0, 1, 0, -1)
CZ = (0, 0, 0, 0, 0, 0, 0, 0, 0, 1, 1, 1, 1, 1, -1, -1, -1, -1, -1)
C = list(zip(CX, CY, CZ))
OPP = [C.index((-x, -y, -z)) for x, y, z in C]
W = [1 / 3 if c == (0, 0, 0) else 1 / 18 if sum(map(abs, c)) == 1 else 1 / 36 for c in C]
STRESS = (9, 11, 13, 14, 15)


def _t(v):
    return torch.tensor(v, dtype=torch.float64, device=DEV)


@functools.lru_cache(maxsize=1)
def _basis():
    """the 19 moments of the MRT models as polynomials of the velocities, and the way back"""
    rows = [[] for _ in range(19)]
    for x, y, z in C:
        c2 = x * x + y * y + z * z
        xx, ww = 3 * x * x - c2, y * y - z * z
        for r, v in zip(rows, (1, 19 * c2 - 30, (21 * c2 * c2 - 53 * c2 + 24) / 2, x, (5 * c2 - 9) * x, y,
                               (5 * c2 - 9) * y, z, (5 * c2 - 9) * z, xx, (3 * c2 - 5) * xx, ww, (3 * c2 - 5) * ww,
                               x * y, y * z, x * z, (y * y - z * z) * x, (z * z - x * x) * y, (x * x - y * y) * z)):
            r.append(v)
    M = _t(rows)
    return M, M.T / (M * M).sum(1)   # its rows are orthogonal


def _meq(model, rho, j):
    """the 19 equilibrium moments at density rho and momentum j[3]"""
    x, y, z = j
    q = x * x + y * y + z * z
    o = torch.zeros_like(rho)
    a, b = 2 * x * x - (y * y + z * z), y * y - z * z
    di3 = model == "MRT_DI3"
    return torch.stack([rho, -11 * rho + 19 * q, 3 * rho - 5.5 * q if di3 else 7.53968254 * q, x, -0.666666667 * x, y,
                        -0.666666667 * y, z, -0.666666667 * z, a, -0.5 * a * 0.333333333333 if di3 else o, b,
                        -0.5 * b if di3 else o, x * y, y * z, x * z, o, o, o])


def _bgk_eq(rho, j):
    q = j[0] * j[0] + j[1] * j[1] + j[2] * j[2]
    return torch.stack([w * (rho + 3 * cu + 4.5 * cu * cu - 1.5 * q)
                        for w, cu in ((w, c[0] * j[0] + c[1] * j[1] + c[2] * j[2]) for w, c in zip(W, C))])


def _equilibrium(model, rho, j):
    if model == "BGK":
        return _bgk_eq(rho, j)
    m = _meq(model, rho, j)
    return (_basis()[1] @ m.reshape(19, -1)).reshape(m.shape)


def _moments(f):
    c = _t(C).T
    j = (c @ f.reshape(19, -1)).reshape((3,) + f.shape[1:])
    return f.sum(0), j


def _pi_neq(f, rho, j):
    p = []
    for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)):
        w = _t([c[a] * c[b] for c in C])
        v = (w[None] @ f.reshape(19, -1)).reshape(f.shape[1:]) - j[a] * j[b]
        p.append(v - rho / 3 if a == b else v)
    return p


def _features(p, tau0):
    xx, yy, zz, xy, xz, yz = p
    pp = xx * xx + yy * yy + zz * zz + 2 * (xy * xy + xz * xz + yz * yz)
    tr3 = (xx ** 3 + yy ** 3 + zz ** 3 + 3 * xx * (xy * xy + xz * xz) + 3 * yy * (xy * xy + yz * yz) +
           3 * zz * (xz * xz + yz * yz) + 6 * xy * xz * yz)
    x = torch.zeros(pp.shape + (16,), dtype=torch.float64, device=DEV)
    x[..., 12] = torch.sqrt(2 * pp) / P_REF
    x[..., 13] = torch.where(pp > 1e-30, tr3 / torch.clamp(pp, min=1e-300) ** 1.5, torch.zeros_like(pp))
    x[..., 14] = (tau0 - 0.5) * 100
    x[..., 15] = 1.0
    return x


def _split(params):
    p = torch.as_tensor(params, device=DEV).double()
    w1, w2, b2, w3, b3 = torch.split(p, [1024, 4096, 64, 64, 1])
    return w1.reshape(64, 16), w2.reshape(64, 64), b2, w3, b3


def _forward(net, X):
    """h1, h2 and the pre-activation of the output; hidden unit 63 is the constant 1"""
    w1, w2, b2, w3, b3 = net
    h1 = torch.relu(X @ w1.T)
    h1[:, 63] = 1.0
    h2 = torch.relu(h1 @ w2.T + b2)
    return h1, h2, h2 @ w3 + b3


def _coefficient(net, X):
    return torch.cat([NU_SCALE * torch.nn.functional.softplus(_forward(net, x)[2]) for x in X.split(1 << 20)])


def _collide(model, f, tau0, les, nu=None, net=None):
    """the collision; nu: the closure's eddy viscosity, or net: evaluate it.  Returns f and that viscosity"""
    rho, j = _moments(f)
    tau = torch.full_like(rho, tau0)
    if net is not None:
        x = _features([-1.5 * v / rho for v in _pi_neq(f, rho, j)], tau0)
        nu = _coefficient(net, x.reshape(-1, 16)).reshape(rho.shape) * x[..., 12] / tau0
    if nu is not None:
        tau = tau0 + 3 * nu
    elif les:
        p = _pi_neq(f, rho, j)
        q = torch.sqrt(p[0] ** 2 + p[1] ** 2 + p[2] ** 2 + 2 * (p[3] ** 2 + p[4] ** 2 + p[5] ** 2))
        tau = 0.5 * tau0 + 0.5 * torch.sqrt(tau0 * tau0 + 18 * math.sqrt(2.0) * 0.01 * q)
    if model == "BGK":
        return f - (f - _bgk_eq(rho, j)) / tau, nu
    M, inv = _basis()
    eq = _meq(model, rho, j)
    m = (M @ f.reshape(19, -1)).reshape(f.shape)
    post = eq.clone()
    for k in STRESS:
        post[k] = m[k] - (m[k] - eq[k]) / tau
    post = (inv @ post.reshape(19, -1)).reshape(f.shape)
    return post, nu


def _lid(f, u):
    """the regularised moving lid on z = nz - 1 (density from the known populations)"""
    rho = sum(f[q] for q in range(19) if CZ[q] == 0) + 2 * sum(f[q] for q in range(19) if CZ[q] > 0)
    j = torch.stack([torch.full_like(rho, u), torch.zeros_like(rho), torch.zeros_like(rho)])
    fe = _bgk_eq(rho, j)
    g = f - fe
    g = torch.stack([g[OPP[q]] if CZ[q] < 0 else g[q] for q in range(19)])
    P = {(a, b): sum(c[a] * c[b] * g[q] for q, c in enumerate(C)) for a in range(3) for b in range(3)}
    tr = (P[0, 0] + P[1, 1] + P[2, 2]) / 3
    return torch.stack([fe[q] + 4.5 * W[q] * (sum(c[a] * c[b] * P[a, b] for a in range(3) for b in range(3)) - tr)
                        for q, c in enumerate(C)])


def _philox(seed, cell, step):
    """Philox4x32-10 of counter (cell, step, 0, 0) and key (seed, 0) as a float in [0, 1)"""
    lo = np.uint64(0xFFFFFFFF)
    c = [cell.astype(np.uint64), np.full(cell.shape, step, np.uint64), np.zeros(cell.shape, np.uint64),
         np.zeros(cell.shape, np.uint64)]
    k0, k1 = seed & 0xFFFFFFFF, 0
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & lo, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & lo]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return (c[0] >> np.uint64(8)).astype(np.float64) / 16777216.0


def _inlet(f, u):
    """momentum set to (u, 0, 0), every other moment kept"""
    _, j = _moments(f)
    d = torch.stack([u - j[0], -j[1], -j[2]]) * 0.1
    return torch.stack([f[q] + c[0] * d[0] + c[1] * d[1] + c[2] * d[2] for q, c in enumerate(C)])


def _outlet(f):
    return f + (1.0 - f.sum(0)) / 19


def _pull(f):
    return torch.stack([torch.roll(f[q], (CZ[q], CY[q], CX[q]), (0, 1, 2)) for q in range(19)])


def _flow_solid(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    z, y, x = torch.meshgrid(torch.arange(nz, device=DEV), torch.arange(ny, device=DEV), torch.arange(nx, device=DEV),
                             indexing="ij")
    if case["geometry"] == "cavity":
        return (((x == 0) | (x == nx - 1) | (y == 0) | (y == ny - 1) | (z == 0)) & (z != nz - 1))
    cx, cy, r = _body(case)
    dx, dy = x - cx, y - cy
    body = (dx.abs() < r) & (dy.abs() < r) if case["geometry"] == "channel_square" else dx * dx + dy * dy < r * r
    inside = (x > 0) & (x < nx - 1)
    return (body & inside) | (y == 0) | (y == ny - 1)


def _exact_flow(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["refined"] or nx * ny * nz * case["steps"] > 1.0e9:
        return None
    cavity = case["geometry"] == "cavity"
    f = _start(case["model"], (nz, ny, nx), 0.0 if cavity else 0.05, seed).double()
    solid = _flow_solid(case)
    source = [torch.roll(solid, (c[2], c[1], c[0]), (0, 1, 2)) & ~solid for c in C]
    tau0 = 1 / float(np.float32(1) / np.float32(case["tau"]))
    net = _split(_weights()) if case["closure_every"] else None
    cell = (np.arange(nz)[:, None] * ny + np.arange(ny)[None]) * nx
    nu, stats, half = None, torch.zeros((4, nz, ny, nx), dtype=torch.float64, device=DEV), max(1, case["steps"] // 2)
    inner = slice(1, ny - 1)
    for t in range(case["steps"]):
        g = _pull(f)
        if case["halfway"]:
            for q in range(1, 19):
                g[q] = torch.where(source[q], f[OPP[q]], g[q])
        if cavity:
            g[:, -1] = _lid(g[:, -1], 0.05)
        else:
            u = torch.full((nz, ny), 0.05, dtype=torch.float64, device=DEV)
            if case["noise"]:
                u = u * (1 + 0.01 * (2 * torch.from_numpy(_philox(seed % 1_000_003, cell, t)).to(DEV) - 1))
            g[:, :, inner, 0] = _inlet(f[:, :, inner, 1], u[:, inner])
            g[:, :, inner, -1] = _outlet(f[:, :, inner, -2])
        fresh = net if case["closure_every"] and t % case["closure_every"] == 0 else None
        post, nu = _collide(case["model"], g, tau0, case["les"], nu if fresh is None else None, fresh)
        f = torch.where(solid, g[OPP], post)
        if case["stats"]:
            j = _moments(f)[1]
            for k in range(2):
                if t < half:
                    stats[k] = torch.where(solid, 0.0, (stats[k] * t + j[k]) / (t + 1))
                else:
                    d = (j[k] - stats[k]) ** 2
                    stats[2 + k] = torch.where(solid, 0.0, (stats[2 + k] * (t - half) + d) / (t - half + 1))
    got = {"f0": f}
    if case["stats"]:
        got["stats"] = stats
    return got


def _exact_calls(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    f = _start(case["model"], (nz, ny, nx), 0.05, seed).double()
    m = _calls_mask(case)[..., :nx]
    body, solid = m == lbm.NODE["BODY"], (m == lbm.NODE["BODY"]) | (m == lbm.NODE["WALL"])
    g = _pull(f)
    force = torch.stack([2 * sum(c[a] * g[q] for q, c in enumerate(C))[body].sum() for a in range(3)])
    inner = slice(1, ny - 1)
    g[:, :, inner, 0] = _inlet(f[:, :, inner, 1], 0.05)
    g[:, :, inner, -1] = _outlet(f[:, :, inner, -2])
    tau0 = 1 / float(np.float32(1.0 / case["tau"]))
    out = torch.zeros((19, nz, ny, case["pitch"]), dtype=torch.float64, device=DEV)
    out[..., :nx] = torch.where(solid, g[OPP], _collide(case["model"], g, tau0, case["les"])[0])
    return dict(f=out, force=force)


class _SplitMix:
    """splitmix64, the generator of the ensembles' modes and of the training shuffles"""

    def __init__(self, seed, add):
        self.s = (seed * 0x9E3779B97F4A7C15 + add) & (2 ** 64 - 1)

    def next(self):
        self.s = (self.s + 0x9E3779B97F4A7C15) & (2 ** 64 - 1)
        z = self.s
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & (2 ** 64 - 1)
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & (2 ** 64 - 1)
        return z ^ (z >> 31)

    def uniform(self):
        return (self.next() >> 11) / 9007199254740992.0


@functools.lru_cache(maxsize=None)
def _shell(k):
    """one wavevector of each +-k pair with a length in [k - 1/2, k + 1/2)"""
    r = range(-k - 1, k + 2)
    return [(a, b, c) for a in r for b in r for c in r
            if k - 0.5 <= math.sqrt(a * a + b * b + c * c) < k + 0.5 and (a, b, c) > (0, 0, 0)]


def _mode_count(n):
    return sum(min(24, len(_shell(k))) for k in range(1, max(1, n // 8) + 1))


def _modes(n, seed):
    """random-phase solenoidal modes, E(k) ~ k^(-5/3), scaled to rms 0.04 per component"""
    r, modes = _SplitMix(seed, 0xD1B54A32D192ED03), []
    for k in range(1, max(1, n // 8) + 1):
        shell = list(_shell(k))
        for i in range(len(shell) - 1, 0, -1):
            j = r.next() % (i + 1)
            shell[i], shell[j] = shell[j], shell[i]
        take = min(24, len(shell))
        amp = math.sqrt(4 * k ** (-5 / 3) / take)
        for kv in shell[:take]:
            kk = math.sqrt(sum(a * a for a in kv))
            while True:
                v = [2 * r.uniform() - 1 for _ in range(3)]
                dot = sum(a * b for a, b in zip(v, kv)) / kk
                v = [a - dot * b / kk for a, b in zip(v, kv)]
                if sum(a * a for a in v) >= 1e-6:
                    break
            vn = math.sqrt(sum(a * a for a in v))
            modes.append((kv, 2 * r.uniform(), [amp * a / vn for a in v]))
    s2 = sum(a * a for _, _, v in modes for a in v)
    scale = 0.04 / math.sqrt(s2 / 6)
    return [(kv, ph, [scale * a for a in v]) for kv, ph, v in modes]


def _turbulence(n, seed):
    u = torch.zeros((3, n, n, n), dtype=torch.float64, device=DEV)
    ax = torch.arange(n, device=DEV)
    for kv, ph, v in _modes(n, seed):
        arg = (kv[0] * ax[None, None, :] + kv[1] * ax[None, :, None] + kv[2] * ax[:, None, None]) % n
        c = torch.cos(math.pi * (2.0 * arg.double() / n + ph))
        for i in range(3):
            u[i] += v[i] * c
    return u


def _filtered(u, tau0):
    """features and least-squares eddy viscosity of the 2x2x2-filtered velocity"""
    n = u.shape[1] // 2

    def box(a):
        return a.reshape(a.shape[0], n, 2, n, 2, n, 2).mean(dim=(2, 4, 6))

    ub = box(u)
    pairs = ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))
    tau = box(torch.stack([u[a] * u[b] for a, b in pairs])) - torch.stack([ub[a] * ub[b] for a, b in pairs])
    g = [[0.5 * (torch.roll(ub[k], -1, 2 - d) - torch.roll(ub[k], 1, 2 - d)) for d in range(3)] for k in range(3)]
    S = torch.stack([0.5 * (g[a][b] + g[b][a]) for a, b in pairs])
    tau[:3] -= tau[:3].sum(0) / 3
    w = _t([1, 1, 1, 2, 2, 2])[:, None, None, None]
    ts, ss = (w * tau * S).sum(0), (w * S * S).sum(0)
    shifts = [(i, j, k) for i in (-1, 0, 1) for j in (-1, 0, 1) for k in (-1, 0, 1)]
    ts, ss = (sum(torch.roll(a, s, (0, 1, 2)) for s in shifts) for a in (ts, ss))
    nu = torch.where(ss > 1e-30, torch.clamp(-ts / (2 * torch.clamp(ss, min=1e-300)), min=0.0), torch.zeros_like(ss))
    return _features(list((tau0 + 3 * nu) * S), tau0).reshape(-1, 16), nu.reshape(-1)


def _exact_boxes(case, seed):
    sizes, tau = _sizes(case), float(np.float32(_box_tau(case)))
    if sum(n ** 3 for n in sizes) * case["steps"] > 1.6e9:
        return None
    net = _split(_weights()) if case["sgs"] == "mlp" else None
    us = []
    for m, n in enumerate(sizes):
        if case["sgs"] == "none":
            u = _turbulence(n, ((seed % 1_000_003) << 8) + m)
            f = _bgk_eq(torch.ones_like(u[0]), u)
        else:
            f = _box_start(n, m, seed).double()
        for _ in range(case["steps"]):
            f, _ = _collide("MRT", _pull(f), tau, case["sgs"] == "smagorinsky", None, net)
        rho, j = _moments(f)
        us.append(j / rho)
    if case["sgs"] != "none":
        return us
    got = [_filtered(u, float(np.float32(0.505))) for u in us]
    return dict(energy=torch.stack([0.5 * (u * u).sum() / u[0].numel() for u in us]),
                X=torch.cat([x for x, _ in got]), T=torch.cat([t for _, t in got]))


def _gradient(net, X, T):
    """gradient (parameter order) and mean of the squared error of o / NU_SCALE"""
    _, w2, _, w3, _ = net
    n = X.shape[0]
    got, loss = [0.0] * 5, 0.0
    for x, t in zip(X.split(1 << 18), T.split(1 << 18)):
        h1, h2, y = _forward(net, x)
        err = torch.nn.functional.softplus(y) - t / NU_SCALE
        loss = loss + (err * err).sum() / n
        dy = 2 * err / n * torch.sigmoid(y)
        d2 = dy[:, None] * w3 * (h2 > 0)
        d1 = (d2 @ w2) * (h1 > 0)
        d1[:, 63] = 0.0
        for k, v in enumerate((d1.T @ x, d2.T @ h1, d2.sum(0), h2.T @ dy, dy.sum()[None])):
            got[k] = got[k] + v
    return torch.cat([v.reshape(-1) for v in got]), loss


def _exact_fit(case, seed):
    n, batch = case["n"], case["batch"]
    X, T = (v.double() for v in _samples(n, seed))
    p = torch.as_tensor(_fresh_params(seed), device=DEV).double()
    m, v, loss = torch.zeros_like(p), torch.zeros_like(p), []
    r, perm, pos = _SplitMix(seed % 1_000_003, 0x632BE59BD9B4E019), list(range(n)), n
    lr, b1, b2, eps = (float(np.float32(a)) for a in (2e-3, 0.9, 0.999, 1e-8))
    for step in range(1, case["steps"] + 1):
        if pos + batch > n:
            for i in range(n - 1, 0, -1):
                k = r.next() % (i + 1)
                perm[i], perm[k] = perm[k], perm[i]
            pos = 0
        at = torch.tensor(perm[pos:pos + batch], device=DEV)
        g, e = _gradient(_split(p), X[at], T[at])
        loss.append(e)
        m, v = b1 * m + (1 - b1) * g, b2 * v + (1 - b2) * g * g
        p = p - lr * (m / (1 - b1 ** step)) / (torch.sqrt(v / (1 - b2 ** step)) + eps)
        pos += batch
    return dict(params=p, loss=torch.stack(loss))


def _exact_evaluate(case, seed):
    X, T = (v.double() for v in _samples(case["n"], seed))
    net = _split(_weights() + np.float32(0.02) * _fresh_params(seed))
    grad, loss = _gradient(net, X, T)
    o = _coefficient(net, X)
    return dict(grad=grad, loss=loss[None], o=o, o_tc=o)


def exact(case, seed):
    return {"flow": _exact_flow, "calls": _exact_calls, "boxes": _exact_boxes, "fit": _exact_fit,
            "evaluate": _exact_evaluate}[case["kind"]](case, seed)
