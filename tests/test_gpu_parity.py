"""GPU parity tests: the CUDA path through the C ABI against the oracle, and
against the golden fixtures the reference's own kernels produced.

Gates (FP32): velocity relative L2 <= 1e-5 after the run (the north-star
gate), drag/lift relative L2 <= 1e-4; FP16 / BF16 storage against the FP64
twin as stated at test_storage_precision_vs_fp64.
"""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from oracle_bindings import CX, CY, CZ, REF_CODE, OracleRun, Refine, moments, rel_l2

pytestmark = pytest.mark.gpu

RTOL = 1e-5
# drag/lift: the gate is on velocity; the force history of the BGK and
# tau0 ~ 0.51 runs amplifies FP32 rounding to ~1e-5, so forces get 1e-4
FTOL = 1e-4
NX, NY, NZ = 64, 24, 6


def _fluid(mask):
    return (mask != 1) & (mask != 2)


def _chan_inputs(lbm, steps, **kw):
    args = dict(obst1=(20.5, 11.5, 0.0), r1=4.0, re=60.0, umax=0.05, tmax=steps, les=1, cs=0.01,
                geometry="channel_square")
    args.update(kw)
    return lbm.make_inputs(NX, NY, NZ, **args)


def _compare(f_gpu, f_orc, mask):
    fl = _fluid(mask)
    rg, jg = moments(f_gpu)
    ro, jo = moments(f_orc)
    return rel_l2(jg[:, fl], jo[:, fl]), float(np.abs(rg[fl] - ro[fl]).max())


@pytest.mark.parametrize("model,les,re,dpdy", [("MRT", 1, 60.0, None), ("MRT", 0, 12.0, None),
                                                ("BGK", 1, 60.0, None), ("MRT_DI3", 1, 60.0, -2e-6),
                                                ("MRT_CPU3D", 0, 12.0, None)])
def test_channel_vs_oracle(product, model, les, re, dpdy):
    lbm = product
    steps = 200
    with lbm.Solver(_chan_inputs(lbm, steps, model=model, les=les, re=re, dpdy=dpdy)) as s:
        s.step(steps)
        f, mask, om, F = s.populations(), s.mask(), s.params()["omega"], s.forces()
    o = OracleRun(NX, NY, NZ, mask, om, model=lbm.MODELS[model], les=les, cs=0.01, dpdy=dpdy or 0.0,
                  init_kind=1 if model == "BGK" else 0, init_u=0.05)
    o.step(steps)
    err, drho = _compare(f, o.fa, mask)
    assert err < RTOL and drho < 1e-5, (err, drho)
    assert rel_l2(F[:, 0], np.array(o.forces)[: len(F), 0]) < FTOL


@pytest.mark.parametrize("name", ["chan_les", "chan_mrt", "chan_les_1k"])
def test_channel_vs_reference_kernels(product, golden, name):
    """the CUDA path against the fields the reference's own kernels produced
    (chan_les_1k: the MRT-LES channel after 1000 steps, the 1e-5 gate)"""
    lbm = product
    meta = golden["meta"][name]
    want = golden["runs"][f"{name}_fields"]
    with lbm.Solver(meta["inputs"]) as s:
        s.step(meta["steps"])
        f, mask, F = s.populations(), s.mask(), s.forces()
    fl = _fluid(mask)
    rho, j = moments(f)
    assert rel_l2(j[:, fl], want[1:, fl]) < RTOL
    assert np.abs(rho[fl] - want[0][fl]).max() < 1e-5
    Fr = golden["runs"][f"{name}_forces"]
    assert rel_l2(F[: len(Fr), 0], Fr[:, 0]) < FTOL


def _lr_setup(lbm, les=1, re=60.0, steps=100):
    return lbm.make_inputs(64, 24, 4, obst1=(20.5, 11.5, 0.0), r1=3.0, re=re, umax=0.05, tmax=steps, les=les,
                           cs=0.01, refinement=1, lr_dims=(32, 32, 8), lr_factor=0.5, lr_origin=(12.25, 4.25, -0.75),
                           geometry="channel_square")


def test_refinement_vs_reference_kernels(product, golden):
    lbm = product
    meta = golden["meta"]["lr"]
    with lbm.Solver(meta["inputs"]) as s:
        assert s.nlevels == 2
        s.step(meta["steps"])
        fc, ff, mc, mf, F = s.populations(0), s.populations(1), s.mask(0), s.mask(1), s.forces()
    _, jc = moments(fc)
    _, jf = moments(ff)
    wc, wf = golden["runs"]["lr_fields"], golden["runs"]["lr_fine_fields"]
    assert rel_l2(jc[:, _fluid(mc)], wc[1:, _fluid(mc)]) < RTOL
    assert rel_l2(jf[:, mf != 2], wf[1:, mf != 2]) < RTOL
    Fr = golden["runs"]["lr_forces"]
    assert rel_l2(F[: len(Fr), 0], Fr[:, 0]) < FTOL


@pytest.mark.parametrize("les,re", [(1, 60.0), (0, 20.0)])
def test_refinement_vs_oracle(product, les, re):
    lbm = product
    steps = 60
    with lbm.Solver(_lr_setup(lbm, les, re, steps)) as s:
        s.step(steps)
        fc, ff, mc, mf, pr = s.populations(0), s.populations(1), s.mask(0), s.mask(1), s.params()
    r = Refine(cnx=64, cny=24, cnz=4, fnx=32, fny=32, fnz=8, lrx0=12.25, lry0=4.25, lrz0=-0.75, lrfactor=0.5,
               lrlevel=2, order=2, cs=0.01, omega_c=pr["omega"], omega_f=pr["omega_lr"], quirk_fc_top_zflip=1)
    o = OracleRun(64, 24, 4, mc, pr["omega"], les=les, cs=0.01, refine=dict(r=r, mask=mf, omega_f=pr["omega_lr"]))
    o.step(steps)
    assert _compare(fc, o.fa, mc)[0] < RTOL
    _, jf = moments(ff)
    _, jo = moments(o.ffa)
    assert rel_l2(jf[:, mf != 2], jo[:, mf != 2]) < RTOL


def _lr_time_setup(lbm, steps):
    return _lr_setup(lbm, 1, 60.0, steps).replace("GPUs per node \t: 1\n", "GPUs per node \t: 1\nCF TIME: \tlinear\n")


def test_refinement_temporal_interpolation_vs_oracle(product):
    """CF TIME: linear (an extension; the reference fills the fine band once
    per coarse step): before the second fine sub-step the band gets the
    coarse moments halfway between the previous and the current coarse
    export.  Against the oracle's loop doing the same; and not the
    reference schedule's result"""
    lbm = product
    steps = 60
    text = _lr_time_setup(lbm, steps)
    assert "CF TIME: \tlinear" in lbm.normalize_inputs(text)
    with lbm.Solver(text) as s:
        s.step(steps)
        fc, ff, mc, mf, pr = s.populations(0), s.populations(1), s.mask(0), s.mask(1), s.params()
    with lbm.Solver(_lr_setup(lbm, 1, 60.0, steps)) as s0:
        s0.step(steps)
        ff0 = s0.populations(1)
    r = Refine(cnx=64, cny=24, cnz=4, fnx=32, fny=32, fnz=8, lrx0=12.25, lry0=4.25, lrz0=-0.75, lrfactor=0.5,
               lrlevel=2, order=2, cs=0.01, omega_c=pr["omega"], omega_f=pr["omega_lr"], quirk_fc_top_zflip=1)
    o = OracleRun(64, 24, 4, mc, pr["omega"], les=1, cs=0.01, refine=dict(r=r, mask=mf, omega_f=pr["omega_lr"]),
                  cf_time=True)
    o.step(steps)
    assert _compare(fc, o.fa, mc)[0] < RTOL
    _, jf = moments(ff)
    _, jo = moments(o.ffa)
    assert rel_l2(jf[:, mf != 2], jo[:, mf != 2]) < RTOL
    _, j0 = moments(ff0)
    assert rel_l2(jf[:, mf != 2], j0[:, mf != 2]) > 100 * RTOL


@pytest.mark.parametrize("cf_time", ["none", "linear"])
def test_z_bounded_patch_vs_oracle(product, cf_time):
    """a fine patch bounded in z (an extension; the reference's spans the
    periodic z extent): 32x32x12 fine from coarse z = 2.25 in a 64x24x12
    channel, the band also on its bottom and top planes and the restriction
    with a z margin too; against the oracle, with and without linear temporal
    interpolation"""
    lbm = product
    steps = 50
    text = lbm.make_inputs(64, 24, 12, obst1=(20.5, 11.5, 0.0), r1=3.0, re=60.0, umax=0.05, tmax=steps, les=1,
                           cs=0.01, refinement=1, lr_dims=(32, 32, 12), lr_factor=0.5, lr_origin=(12.25, 4.25, 2.25),
                           geometry="channel_square", cf_time=cf_time)
    with lbm.Solver(text) as s:
        s.step(steps)
        fc, ff, mc, mf, pr = s.populations(0), s.populations(1), s.mask(0), s.mask(1), s.params()
    assert np.isfinite(ff).all()
    r = Refine(cnx=64, cny=24, cnz=12, fnx=32, fny=32, fnz=12, lrx0=12.25, lry0=4.25, lrz0=2.25, lrfactor=0.5,
               lrlevel=2, order=2, cs=0.01, omega_c=pr["omega"], omega_f=pr["omega_lr"], quirk_fc_top_zflip=1,
               zbounded=1, cz0=2)
    o = OracleRun(64, 24, 12, mc, pr["omega"], les=1, cs=0.01, refine=dict(r=r, mask=mf, omega_f=pr["omega_lr"]),
                  cf_time=cf_time == "linear")
    o.step(steps)
    assert _compare(fc, o.fa, mc)[0] < RTOL
    _, jf = moments(ff)
    _, jo = moments(o.ffa)
    assert rel_l2(jf[:, mf != 2], jo[:, mf != 2]) < RTOL


@pytest.mark.parametrize("cf_time", ["none", "linear"])
def test_patch_of_ratio_4_vs_oracle(product, cf_time):
    """four fine sub-steps per coarse step: the band filled before each of the
    middle ones and, with the end of the coarse step, before the last"""
    lbm = product
    steps = 12
    text = lbm.make_inputs(64, 24, 12, obst1=(20.5, 11.5, 0.0), r1=2.0, re=30.0, umax=0.05, tmax=steps, les=1,
                           cs=0.01, refinement=1, lr_dims=(48, 40, 24), lr_factor=0.25, lr_origin=(15.125, 6.125, 2.125),
                           geometry="channel_square", cf_time=cf_time)
    with lbm.Solver(text) as s:
        s.step(steps)
        fc, ff, mc, mf, pr = s.populations(0), s.populations(1), s.mask(0), s.mask(1), s.params()
    assert np.isfinite(ff).all()
    r = Refine(cnx=64, cny=24, cnz=12, fnx=48, fny=40, fnz=24, lrx0=15.125, lry0=6.125, lrz0=2.125, lrfactor=0.25,
               lrlevel=4, order=2, cs=0.01, omega_c=pr["omega"], omega_f=pr["omega_lr"], quirk_fc_top_zflip=1,
               zbounded=1, cz0=2)
    o = OracleRun(64, 24, 12, mc, pr["omega"], les=1, cs=0.01, refine=dict(r=r, mask=mf, omega_f=pr["omega_lr"]),
                  cf_time=cf_time == "linear")
    o.step(steps)
    assert _compare(fc, o.fa, mc)[0] < RTOL
    _, jf = moments(ff)
    _, jo = moments(o.ffa)
    assert rel_l2(jf[:, mf != 2], jo[:, mf != 2]) < RTOL


@pytest.mark.parametrize("cf_time", ["none", "linear"])
def test_refinement_step_graphs_are_bit_exact(product, cf_time):
    """lbm_step captures refinement steps in batches into CUDA graphs; one
    call of n steps (one direct step, then batches of 16, 16 and 7 replayed
    from graphs) equals n calls of one step (launched directly) bit for bit
    on both levels, with
    running statistics and inlet noise on (both take the step index baked
    into each captured launch), with and without linear temporal
    interpolation"""
    lbm = product
    steps = 40
    text = lbm.make_inputs(128, 48, 8, obst1=(40.5, 23.5, 0.0), r1=3.0, re=60.0, umax=0.05, tmax=steps, les=1,
                           cs=0.01, refinement=1, lr_dims=(48, 48, 16), lr_factor=0.5, lr_origin=(28.25, 12.25, -0.75),
                           geometry="channel_square", cf_time=cf_time, velav=1, start_velav=10, start_velfluc=25,
                           inlet_noise=0.01, seed=7)
    with lbm.Solver(text) as a:
        a.step(steps)
        fa = [a.populations(0), a.populations(1)]
        sa = [a.stats(0), a.stats(1)]
    with lbm.Solver(text) as b:
        for _ in range(steps):
            b.step(1)
        fb = [b.populations(0), b.populations(1)]
        sb = [b.stats(0), b.stats(1)]
    assert np.isfinite(fa[1]).all() and np.abs(sa[0]).max() > 0
    for x, y in zip(fa + sa, fb + sb):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("precision", ["fp32", "fp16"])
def test_uniform_step_graphs_are_bit_exact(product, precision):
    """the same for a uniform channel: 40 steps in one call (graphs of 16,
    16 and 8 steps, the drag/lift reduction forked to the side stream and
    joined inside each step) against 40 single steps: populations,
    statistics and the per-step force history bit for bit"""
    lbm = product
    steps = 40
    text = _chan_inputs(lbm, steps, velav=1, start_velav=10, start_velfluc=25, inlet_noise=0.01, seed=3,
                        precision=precision, bounceback="halfway")
    with lbm.Solver(text) as a:
        a.step(steps)
        ra = [a.populations(), a.stats(), a.forces(steps)]
    with lbm.Solver(text) as b:
        for _ in range(steps):
            b.step(1)
        rb = [b.populations(), b.stats(), b.forces(steps)]
    assert np.abs(ra[2]).max() > 0
    for x, y in zip(ra, rb):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("kind", ["stats_noise", "no_body", "fp16_late_force", "refined", "new_mask",
                                  "closure_5", "closure_16"])
def test_replayed_step_graphs_are_bit_exact(product, kind):
    """graphs launched again without a new capture (the step number on the
    device): calls of several lengths equal single steps in populations,
    statistics and the recorded forces, with statistics and inlet noise, with
    no body, with the force recorded from a later step on, with refinement,
    with the mask changed in between, and with the learned closure evaluated
    every 5 or 16 steps"""
    lbm = product
    kw = dict(obst1=(18.5, 11.5, 0.0), r1=4.0, re=60.0, umax=0.05, tmax=400, les=1, cs=0.01, bounceback="halfway",
              inlet_noise=0.01, seed=5)
    if kind == "stats_noise":
        kw.update(velav=1, start_velav=20, start_velfluc=70)
    elif kind == "no_body":
        kw.update(geometry="channel")
    elif kind == "fp16_late_force":
        kw.update(precision="fp16", startf=37)
    elif kind == "refined":
        kw.update(refinement=1, lr_dims=(32, 32, 12), lr_factor=0.5, lr_origin=(12.25, 4.25, 2.25), cf_time="linear",
                  bounceback="fullway")
    elif kind.startswith("closure"):
        kw.update(sgs="mlp", sgs_every=int(kind[8:]))
    text = lbm.make_inputs(64, 24, 12, **kw)
    res = []
    for calls in ([16, 16, 5, 33, 16, 1, 48], [1] * 135):
        with lbm.Solver(text) as s:
            if kind.startswith("closure"):
                s.set_sgs_mlp(np.fromfile(lbm.LIB_PATH.parent.parent / "data" / "sgs_mlp.bin", np.float32))
            t = 0
            for n in calls:
                s.step(n)
                t += n
                if kind == "new_mask" and t == 70:
                    m = s.mask()
                    m[3:6, 15:18, 40:44] = lbm.NODE["BODY"]
                    s.set_mask(m)
            got = [s.populations(k) for k in range(s.nlevels)] + [s.forces()]
            res.append(got + ([s.stats()] if kind == "stats_noise" else []))
    for a, b in zip(*res):
        np.testing.assert_array_equal(a, b)
    assert np.isfinite(res[0][0]).all()


def test_async_force_read_after_graph_steps(product):
    """lbm_get_last_force_async after a graph-replayed lbm_step(n): the copy
    on the force stream waits for the replayed steps, so it reads the same
    value as the synchronous read on the main stream, step after step"""
    torch = pytest.importorskip("torch")

    lbm = product
    with lbm.Solver(_chan_inputs(lbm, 400)) as s:
        out = torch.zeros(3, dtype=torch.float64, pin_memory=True).numpy()
        for _ in range(8):
            s.step(48)
            s.last_force_async(out)
            s.synchronize()
            want = s.last_force()
            assert np.abs(want).max() > 0
            np.testing.assert_array_equal(out, want)


def test_checkpoint_with_temporal_interpolation_is_bit_exact(product, tmp_path):
    """the kept coarse export travels in the checkpoint: a restart continues
    bit for bit"""
    lbm = product
    ck = tmp_path / "lr.ckpt"
    with lbm.Solver(_lr_time_setup(lbm, 60)) as s:
        s.step(20)
        s.save_state(ck)
        s.step(20)
        f0, f1 = s.populations(0), s.populations(1)
    with lbm.Solver.from_state(ck) as r:
        r.step(20)
        np.testing.assert_array_equal(r.populations(0), f0)
        np.testing.assert_array_equal(r.populations(1), f1)


def test_statistics_vs_oracle(product):
    lbm = product
    steps = 200
    with lbm.Solver(_chan_inputs(lbm, steps, start_velav=50, start_velfluc=120, velav=1)) as s:
        s.step(steps)
        st, mask, om = s.stats(), s.mask(), s.params()["omega"]
    o = OracleRun(NX, NY, NZ, mask, om, les=1, cs=0.01, stats=(50, 120))
    o.step(steps)
    fl = _fluid(mask)
    for k in range(4):
        assert rel_l2(st[k][fl], o.st[k][fl]) < 1e-4, k


def test_inlet_noise_vs_oracle(product):
    """seeded Philox noise: same numbers on both sides, so the runs agree"""
    lbm = product
    steps = 100
    with lbm.Solver(_chan_inputs(lbm, steps, inlet_noise=0.01, seed=777)) as s:
        s.step(steps)
        f, mask, om = s.populations(), s.mask(), s.params()["omega"]
    o = OracleRun(NX, NY, NZ, mask, om, les=1, cs=0.01, noise_amp=0.01, seed=777)
    o.step(steps)
    assert _compare(f, o.fa, mask)[0] < RTOL
    o2 = OracleRun(NX, NY, NZ, mask, om, les=1, cs=0.01)
    o2.step(steps)
    assert _compare(o.fa, o2.fa, mask)[0] > 1e-4  # the noise is really there


def test_lid_cavity_bgk_vs_oracle(product):
    """lid-driven cavity: BGK, tau 0.6, lid on the top face moving +x"""
    lbm = product
    n, steps = 32, 200
    text = lbm.make_inputs(n, n, n, umax=0.05, tmax=steps, model="BGK", geometry="cavity", tau=0.6,
                           lid_velocity=(0.05, 0.0, 0.0), lid_face="+z")
    with lbm.Solver(text) as s:
        s.step(steps)
        f, mask, audit = s.populations(), s.mask(), s.audit()
    o = OracleRun(n, n, n, mask, 1 / 0.6, model=2, init_kind=1, init_u=0.0, lid_u=(0.05, 0, 0), lid_face=5)
    o.step(steps)
    err, _ = _compare(f, o.fa, mask)
    assert err < RTOL
    assert np.isfinite(audit).all()


@pytest.mark.parametrize("model,les", [("MRT", 1), ("BGK", 0)])
def test_halfway_bounceback_vs_oracle(product, model, les):
    """half-way bounce-back (the channel configuration's wall treatment; the
    reference is full-way): velocity and the link-wise drag/lift"""
    lbm = product
    steps = 200
    with lbm.Solver(_chan_inputs(lbm, steps, model=model, les=les, bounceback="halfway")) as s:
        s.step(steps)
        f, mask, om, F = s.populations(), s.mask(), s.params()["omega"], s.forces()
    o = OracleRun(NX, NY, NZ, mask, om, model=lbm.MODELS[model], les=les, cs=0.01,
                  init_kind=1 if model == "BGK" else 0, init_u=0.05, halfway=1)
    o.step(steps)
    err, drho = _compare(f, o.fa, mask)
    assert err < RTOL and drho < 1e-5, (err, drho)
    Fo = np.array(o.forces)[: len(F)]
    assert rel_l2(F[:, 0], Fo[:, 0]) < FTOL and F[-1, 0] > 0
    with lbm.Solver(_chan_inputs(lbm, steps, model=model, les=les)) as s:
        s.step(steps)
        F_full = s.forces()
    assert abs(F_full[-1, 0] - F[-1, 0]) > 1e-3 * abs(F[-1, 0])   # a different wall position, a different drag


@pytest.mark.parametrize("fixture", ["cpu3d_cavity24.npz", "cpu3d_cavity24_1k.npz"])
def test_reference_cpu_program_cavity(product, golden, fixture):
    """CPU_3D semantics on the GPU against the reference CPU program's output
    (100 and 1000 steps)"""
    lbm = product
    d = np.load(golden["dir"] / fixture)
    n = 24
    text = lbm.make_inputs(n, n, n, r1=5.0, re=50.0, umax=0.04, model="MRT_CPU3D", geometry="cavity", lid_face="-x",
                           lid_velocity=(0.0, 0.04, 0.0), init=2, init_velocity=0.04, edge_pull="clamp",
                           lid_bc="cpu3d")
    with lbm.Solver(text) as s:
        s.step(int(d["steps"]))
        f = s.populations()
    rho, j = moments(f)
    assert rel_l2(j[:2], d["uvrho"][:2]) < 1e-5
    assert np.abs(rho - d["uvrho"][2]).max() < 2e-5


def _c1(lbm, n, steps, face, lid_u):
    return lbm.make_inputs(n, n, n, umax=0.05, tmax=steps, model="BGK", geometry="cavity", tau=0.6,
                           lid_velocity=lid_u, lid_face=face)


def test_c1_cavity_64_vs_oracle_and_mass(product):
    """BGK lid-driven cavity 64^3, tau 0.6, lid on the top face moving +x,
    equilibrium start at rest, 1000 steps"""
    lbm = product
    n, steps = 64, 1000
    with lbm.Solver(_c1(lbm, n, steps, "+z", (0.05, 0.0, 0.0))) as s:
        m0 = s.audit()[0]
        s.step(steps)
        f, mask, m1 = s.populations(), s.mask(), s.audit()[0]
    o = OracleRun(n, n, n, mask, 1 / 0.6, model=2, init_kind=1, init_u=0.0, lid_u=(0.05, 0, 0), lid_face=5)
    o.step(steps)
    assert _compare(f, o.fa, mask)[0] < RTOL
    _, j = moments(f)
    assert j[0].max() > 0.01 and np.isfinite(f).all()   # the lid drives the flow
    assert abs(m1 - m0) / m0 < 1e-3


def test_c1_cavity_axis_permutation(product):
    """the same cavity in CPU_3D's orientation (lid at x = 0 moving +y) is the
    axis-permuted image: x' = n-1-z, y' = x, z' = y"""
    lbm = product
    n, steps = 64, 300
    with lbm.Solver(_c1(lbm, n, steps, "+z", (0.05, 0.0, 0.0))) as s:
        s.step(steps)
        _, ja = moments(s.populations())
    with lbm.Solver(_c1(lbm, n, steps, "-x", (0.0, 0.05, 0.0))) as s:
        s.step(steps)
        _, jb = moments(s.populations())
    # jb[c][z', y', x'] with x' = n-1-z, y' = x, z' = y  ->  index jb[:, y, x, n-1-z]
    jbp = jb[:, :, :, ::-1]              # [c][y][x][z]
    jbp = np.transpose(jbp, (0, 3, 1, 2))  # [c][z][y][x]
    mapped = np.stack([jbp[1], jbp[2], -jbp[0]])
    assert rel_l2(mapped, ja) < 1e-5


# FP16 / BF16 store f minus the model's equilibrium at the inlet velocity;
# on this small channel (tau0 0.515, 200 steps) the velocity error against
# the FP64 twin was 1.4e-3 (FP16) and 3.5e-2 (BF16) with the BGK
# equilibrium as the offset, which leaves LR7's m2 (no density term) in the
# stored values
@pytest.mark.parametrize("prec,tol", [("fp16", 2e-3), ("bf16", 5e-2), ("fp32", 1e-5)])
def test_storage_precision_vs_fp64(product, prec, tol):
    lbm = product
    steps = 200
    out = {}
    for p in (prec, "fp64"):
        with lbm.Solver(_chan_inputs(lbm, steps, precision=p)) as s:
            s.step(steps)
            out[p] = (s.populations(), s.mask())
    f, mask = out[prec]
    f64, _ = out["fp64"]
    err, _ = _compare(f, f64, mask)
    assert err < tol, err


def test_mass_conservation_periodic_fp64_audit(product):
    """a fully periodic box conserves mass and momentum exactly; the FP64
    audit sees only FP32 rounding"""
    lbm = product
    n = 48
    with lbm.Solver(lbm.make_inputs(n, n, n, umax=0.05, tmax=10, les=1, cs=0.01, geometry="periodic", tau=0.55,
                                    init_velocity=0.02)) as s:
        a0 = s.audit()
        s.step(300)
        a1 = s.audit()
    assert abs(a1[0] - a0[0]) / a0[0] < 1e-6
    assert abs(a1[1] - a0[1]) / a0[1] < 1e-5


def test_deterministic_runs(product):
    lbm = product
    text = _chan_inputs(lbm, 50, inlet_noise=0.01)
    res = []
    for _ in range(2):
        with lbm.Solver(text) as s:
            s.step(50)
            res.append((s.populations(), s.forces()))
    np.testing.assert_array_equal(res[0][0], res[1][0])
    np.testing.assert_array_equal(res[0][1], res[1][1])


def test_force_side_stream_and_launch_count(product):
    """the per-step force runs on a side stream beside the stream-collide:
    every step's force read asynchronously equals the recorded history, the
    history equals a run that reads it synchronously after each step, and a
    step is exactly two kernels (force + stream-collide; the first step,
    t = STARTF = 0, records no force)"""
    lbm = product
    steps = 40
    text = _chan_inputs(lbm, steps)
    with lbm.Solver(text) as s:
        n0 = s.launch_count()
        got = np.zeros((steps, 3))
        for i in range(steps):
            s.step(1)
            s.last_force_async(got[i])
        s.synchronize()
        assert s.launch_count() - n0 == 2 * steps - 1
        hist = s.forces()
    with lbm.Solver(text) as s:
        sync = np.zeros((steps, 3))
        for i in range(steps):
            s.step(1)
            sync[i] = s.last_force()
    np.testing.assert_array_equal(got, hist[:steps])
    np.testing.assert_array_equal(got, sync)
    assert np.abs(got[-1, 0]) > 0


def test_kernel_level_api_matches_handle(product):
    """lbm_stream_collide_f32 / lbm_body_force_f32 on caller-owned device
    buffers give the handle's step and force"""
    torch = pytest.importorskip("torch")
    lbm = product
    lib = lbm.library()
    with lbm.Solver(_chan_inputs(lbm, 10)) as s:
        f0, mask, om = s.populations(), s.mask(), s.params()["omega"]
        s.step(2)
        f_ref, F_ref = s.populations(), s.forces()
    pitch = 64
    dev = torch.device("cuda", torch.cuda.current_device())
    fa = torch.zeros((19, NZ, NY, pitch), dtype=torch.float32, device=dev)
    fb = torch.zeros_like(fa)
    fa[..., :NX] = torch.from_numpy(f0).to(dev)
    m = torch.full((NZ, NY, pitch), 1, dtype=torch.uint8, device=dev)
    m[..., :NX] = torch.from_numpy(mask).to(dev)
    force = torch.zeros(3, dtype=torch.float64, device=dev)
    scratch = torch.zeros(int(lib.lbm_body_force_scratch_doubles()), dtype=torch.float64, device=dev)
    P = ctypes.c_void_p
    stream = P(torch.cuda.current_stream().cuda_stream)
    for t in range(2):
        if t > 0:
            assert lib.lbm_body_force_f32(P(fa.data_ptr()), P(m.data_ptr()), NX, NY, NZ, pitch, P(force.data_ptr()),
                                          P(scratch.data_ptr()), stream) == 0
        assert lib.lbm_stream_collide_f32(P(fa.data_ptr()), P(fb.data_ptr()), P(m.data_ptr()), NX, NY, NZ, pitch, 0,
                                          1, ctypes.c_float(om), ctypes.c_float(0.01), ctypes.c_float(0.05),
                                          ctypes.c_float(1.0), t, stream) == 0
        fa, fb = fb, fa
    torch.cuda.synchronize()
    np.testing.assert_array_equal(fa[..., :NX].cpu().numpy(), f_ref)
    # same per-node sums, FP64 sums over nodes grouped differently
    assert abs(force[0].item() - F_ref[1, 0]) <= 1e-12 * abs(F_ref[1, 0])


@pytest.mark.parametrize("nx,ny,nz,pitch,shift", [(20, 12, 5, 32, 0), (33, 7, 3, 64, 5), (96, 48, 33, 96, 0),
                                                  (257, 40, 31, 288, 16)])
def test_body_force_scan_against_numpy(product, nx, ny, nz, pitch, shift):
    """the mask scan over scattered and dense bodies, mask buffers off a
    16-byte boundary, domains that end inside a warp's 512 bytes, and BODY
    bytes in the row padding (not part of the domain)"""
    torch = pytest.importorskip("torch")
    lib = product.library()
    rng = np.random.default_rng(nx)
    m = np.zeros((nz, ny, pitch), np.uint8)
    m[rng.random(m.shape) < 0.02] = 2
    m[:, ny // 3:ny // 2, nx // 4:nx // 2] = 2
    m[:, :, nx:] = 2
    f = np.zeros((19, nz, ny, pitch), np.float32)
    f[..., :nx] = rng.random((19, nz, ny, nx), np.float32)
    room = torch.zeros(m.size + shift, dtype=torch.uint8, device="cuda")
    dm = room[shift:].copy_(torch.from_numpy(m.reshape(-1)).cuda())
    df = torch.from_numpy(f).cuda()
    force = torch.zeros(3, dtype=torch.float64, device="cuda")
    scratch = torch.full((int(lib.lbm_body_force_scratch_doubles()),), float("nan"), dtype=torch.float64, device="cuda")
    at = lambda t: ctypes.c_void_p(t.data_ptr())
    assert lib.lbm_body_force_f32(at(df), at(dm), nx, ny, nz, pitch, at(force), at(scratch), None) == 0
    torch.cuda.synchronize()
    g = f[..., :nx].astype(np.float64)
    body = m[..., :nx] == 2
    want, size = np.zeros(3), 0.0
    for q in range(19):
        v = 2 * np.roll(g[q], (CZ[q], CY[q], CX[q]), (0, 1, 2))[body].sum()
        want += np.array([CX[q], CY[q], CZ[q]]) * v
        size += v
    # per node an FP32 sum of 18 terms (18 roundings of 2^-24 each at most), across nodes FP64
    np.testing.assert_allclose(force.cpu().numpy(), want, rtol=0, atol=18 * 2.0 ** -24 * size)


def test_c2_size_properties(product):
    """the 512x128x128 channel: finite, deterministic, mass close to the
    inlet-driven initial state, drag positive"""
    lbm = product
    text = lbm.make_inputs(512, 128, 128, obst1=(128.5, 63.5, 0.0), r1=8.0, re=120.0, umax=0.05, tmax=100, les=1,
                           cs=0.01, geometry="channel_square", inlet_noise=0.01)
    with lbm.Solver(text) as s:
        a0 = s.audit()
        s.step(40)
        a1 = s.audit()
        F = s.forces()
        rho, u, v, w = s.fields()
    assert np.isfinite(rho).all() and np.isfinite(u).all()
    assert abs(a1[0] - a0[0]) / a0[0] < 1e-3
    assert (F[5:, 0] > 0).all()
    assert rho.shape == (128, 128, 512)


def test_output_files_byte_compatible(product, golden, tmp_path):
    """WriteResults / WriteForces / WriteInputs layout: the reference's own
    text for the same populations"""
    import gzip

    lbm = product
    g = golden["dir"]
    text = (g / "writer_tiny.inputs").read_text()
    f = np.load(g / "writer_tiny.npz")["f"]
    with lbm.Solver(text) as s:
        s.set_populations(f)
        s.write_outputs(str(tmp_path / "case"))
        assert s.inputs_text() == text
    zone = (tmp_path / "case_part0.dat").read_text()
    want = gzip.open(g / "writer_tiny_part0.dat.gz", "rt").read()
    # velAv / velFluc columns: statistics are off in this handle, the reference's were on
    cut = lambda t: [",".join(l.split(",")[:7]) for l in t.splitlines()]
    assert cut(zone.rstrip("\n")) == cut(want)
    assert (tmp_path / "case.inputs").read_text() == text


def test_errors_are_reported(product):
    lbm = product
    with pytest.raises(lbm.LbmError) as e:
        lbm.Solver("Base domain size \t64x24x6\nbogus key: \t1\n")
    assert e.value.code == 3 and "unknown key" in str(e.value)
    with pytest.raises(lbm.LbmError) as e:
        lbm.Solver(lbm.make_inputs(64, 24, 4, refinement=1, lr_dims=(32, 32, 6), lr_factor=0.5,
                                   lr_origin=(12.25, 4.25, -0.75)))
    assert e.value.code == 4


@pytest.mark.parametrize("prec", ["fp32", "fp16"])
def test_checkpoint_restart_is_bit_exact(product, tmp_path, prec):
    """stop after 40 steps, restart from the checkpoint, run 40 more: the
    same populations, force history and statistics as never stopping"""
    lbm = product
    text = _chan_inputs(lbm, 100, precision=prec, inlet_noise=0.01, velav=1, start_velav=10, start_velfluc=30,
                        bounceback="halfway")
    ck = tmp_path / "run.ckpt"
    with lbm.Solver(text) as s:
        s.step(40)
        s.save_state(ck)
        s.step(40)
        f1, F1, st1 = s.populations(), s.forces(), s.stats()
    with lbm.Solver.from_state(ck) as r:
        assert r.time == 40
        r.step(40)
        np.testing.assert_array_equal(r.populations(), f1)
        np.testing.assert_array_equal(r.forces(), F1)
        np.testing.assert_array_equal(r.stats(), st1)
    with lbm.Solver(text) as r2:
        r2.step(3)          # any state: the checkpoint replaces it
        r2.restore_state(ck)
        r2.step(40)
        np.testing.assert_array_equal(r2.populations(), f1)
    with lbm.Solver(_chan_inputs(lbm, 100, precision="fp32")) as other:
        if prec != "fp32":
            with pytest.raises(lbm.LbmError):
                other.restore_state(ck)


def test_dynamic_inlet_vs_oracle(product):
    """DI3's dynamic-inlet duct (64x124x20, walls at x = 0 and 63, periodic
    in y and z, DI3 MRT with the body force dpdy below DYNY1): trip blocks
    until t = 50, then the P-control of the plane-mean v every 20 steps after
    t = 60 updates dpdy on the device.  Against the oracle running the same
    loop with the control restated on the host"""
    from oracle_bindings import Params, oracle, ptr

    lbm = product
    nx, ny, nz, steps = 64, 124, 20, 150
    y1, every, start, trip_end, kp, dpdy0, umax = 123, 20, 60, 50, 2.0, -5.16e-7, 0.06
    text = lbm.make_inputs(nx, ny, nz, obst1=(31.5, 92.5, 0.0), r1=31.0, obst2=(25.5, 25.5, 0.0), r2=10.0,
                           re=5400.0, umax=umax, tmax=steps, les=1, cs=0.02, model="MRT_DI3", dpdy=dpdy0,
                           geometry="dyninlet", dyny1=y1, dyn_every=every, dyn_start=start, trip_end=trip_end, kp=kp)
    with lbm.Solver(text) as s:
        om = s.params()["omega"]
        s.step(steps)
        f, mask, hist = s.populations(), s.mask(), s.dyn_history()
    o = oracle()
    m = np.zeros((nz, ny, nx), np.uint8)
    o.orc_mask_dyninlet(ptr(m), nx, ny, nz, ctypes.c_float(25.5), ctypes.c_float(25.5), ctypes.c_float(10.0), 1)
    p = Params(nx=nx, ny=ny, nz=nz, model=1, les=1, omega=om, cs=0.02, dpdy=dpdy0, u_in=umax, rho_out=1.0,
               stats_weight=1.0, dyn_y1=y1)
    fa = np.zeros((19, nz, ny, nx), np.float32)
    o.orc_init_axis(ctypes.byref(p), ptr(m), ptr(fa), 0, ctypes.c_float(umax), 1)
    fb = fa.copy()
    dp = np.float32(dpdy0)
    want = []
    from oracle_bindings import CY
    for t in range(steps):
        if t == trip_end:
            o.orc_mask_dyninlet(ptr(m), nx, ny, nz, ctypes.c_float(25.5), ctypes.c_float(25.5), ctypes.c_float(10.0), 0)
        p.t, p.force_on, p.dpdy = t, 1 if t > 0 else 0, float(dp)
        f3 = np.zeros(3)
        o.orc_step(ctypes.byref(p), ptr(m), ptr(fa), ptr(fb), ptr(f3), None, None, None, None, None)
        fa, fb = fb, fa
        if t % every == 0 and t > start:
            v = np.tensordot(CY.astype(np.float64), fa[:, :, y1, :].astype(np.float64), 1)
            av = np.float32(v.sum() / ((nx - 2) * nz))
            dp = np.float32(dp + np.float32((av - np.float32(umax)) / np.float32(umax)) * np.float32(kp) *
                            np.float32(abs(dpdy0)))
            want.append((t, av, dp))
    want = np.array(want, np.float64)
    assert hist.shape == want.shape and np.array_equal(hist[:, 0], want[:, 0])
    np.testing.assert_allclose(hist[:, 1], want[:, 1], rtol=1e-5)
    np.testing.assert_allclose(hist[:, 2], want[:, 2], rtol=1e-4)
    assert abs(hist[-1, 2] - dpdy0) > 1e-3 * abs(dpdy0)            # the control acted
    err, _ = _compare(f, fa, mask)
    assert err < RTOL


def _alt_bc_mask(case, nx, ny, nz):
    N = lambda k: product_node(k)  # noqa: E731
    m = np.zeros((nz, ny, nx), np.uint8)
    if case == "dirichlet_neumann_ysym":
        m[:, 0, :], m[:, -1, :] = N("YSYM_BOT"), N("YSYM_TOP")
        m[:, :, 0], m[:, :, -1] = N("DIR_WEST"), N("NEU_EAST")
    elif case == "xsym_regularised_zsym":
        m[:, 0, :] = m[:, -1, :] = N("WALL")
        m[0], m[-1] = N("ZSYM_BOT"), N("ZSYM_TOP")
        m[:, 1:-1, 0], m[:, 1:-1, -1] = N("XSYM_BOT"), N("NEU_EAST_REG")
    elif case == "moving_walls_west_v":
        m[:, 0, :], m[:, -1, :] = N("DIR_SOUTH"), N("DIR_NORTH")
        m[:, 1:-1, 0], m[:, 1:-1, -1] = N("DIR_WEST_V"), N("NEU_EAST")
    else:  # "west_reg_xsym_body"
        m[:, 0, :] = m[:, -1, :] = N("WALL")
        m[:, 1:-1, 0], m[:, 1:-1, -1] = N("WEST_REG"), N("XSYM_TOP")
        m[:, 6:10, 12:16] = N("BODY")
    return m


def product_node(k):
    import lbm_multigpu_gb300 as lbm

    return lbm.NODE[k]


@pytest.mark.parametrize("case,model,les", [("dirichlet_neumann_ysym", "MRT_CPU3D", 0),
                                            ("xsym_regularised_zsym", "MRT", 1),
                                            ("west_reg_xsym_body", "BGK", 0),
                                            ("moving_walls_west_v", "MRT", 0)])
def test_alternate_boundaries_vs_oracle(product, case, model, les):
    """the alternate boundary node types (CPU_3D's Dirichlet west, Neumann and
    regularised east, y/z symmetry planes, the tangential west inlet and the
    moving north/south walls; LR7's x symmetry planes; BC1's West_Reg through
    its t = 1000 perturbation) in a 30x16x12 box stepped
    through lbm_stream_collide_f32, against the oracle's step on the same mask"""
    torch = pytest.importorskip("torch")
    lbm = product
    lib = lbm.library()
    nx, ny, nz, pitch, steps, t0, om, u = 30, 16, 12, 32, 80, 960, 1.7, 0.04
    mask = _alt_bc_mask(case, nx, ny, nz)
    # the box starts at half the inlet speed so that the inlet drives the flow
    o = OracleRun(nx, ny, nz, mask, om, model=lbm.MODELS[model], les=les, cs=0.02, u_in=u, init_kind=0,
                  init_u=u / 2)
    o.t = t0
    dev = torch.device("cuda", torch.cuda.current_device())
    fa = torch.zeros((19, nz, ny, pitch), dtype=torch.float32, device=dev)
    fa[..., :nx] = torch.from_numpy(o.fa.copy()).to(dev)
    fb = torch.zeros_like(fa)
    m = torch.full((nz, ny, pitch), 1, dtype=torch.uint8, device=dev)
    m[..., :nx] = torch.from_numpy(mask).to(dev)
    P = ctypes.c_void_p
    stream = P(torch.cuda.current_stream().cuda_stream)
    for t in range(t0, t0 + steps):
        assert lib.lbm_stream_collide_f32(P(fa.data_ptr()), P(fb.data_ptr()), P(m.data_ptr()), nx, ny, nz, pitch,
                                          lbm.MODELS[model], les, ctypes.c_float(om), ctypes.c_float(0.02),
                                          ctypes.c_float(u), ctypes.c_float(1.0), t, stream) == 0
        fa, fb = fb, fa
    torch.cuda.synchronize()
    o.step(steps)
    f = fa[..., :nx].cpu().numpy()
    assert np.isfinite(f).all()
    err, drho = _compare(f, o.fa, mask)
    assert err < RTOL and drho < 1e-5, (err, drho)
    # the boundaries acted: the flow differs from the same box without them
    plain = OracleRun(nx, ny, nz, np.where(mask >= product_node("DIR_WEST"), 0, mask).astype(np.uint8), om,
                      model=lbm.MODELS[model], les=les, cs=0.02, u_in=u, init_kind=0, init_u=u / 2)
    plain.t = t0
    plain.step(steps)
    assert _compare(plain.fa, o.fa, mask)[0] > 100 * RTOL


@pytest.mark.parametrize("faces,model,les", [(None, "MRT_CPU3D", 0),
                                             (("DIR_WEST", "NEU_EAST", "YSYM_BOT", "YSYM_TOP", "ZSYM_BOT",
                                               "ZSYM_TOP"), "MRT", 1)])
def test_duct_solver_vs_oracle(product, faces, model, les):
    """the "duct" geometry through the handle: CPU_3D's cylinder duct with
    its Dirichlet inlet and rho = 1 outlet (walls on y and z), and the same
    duct with symmetry planes from a FACES line; flow and drag/lift against
    the oracle.  (NEU_EAST_REG, NeumannEast_Regularized as the reference
    wrote it, diverges within ~100 steps in such a duct; it is checked per
    cell and in the short box runs only.)"""
    lbm = product
    nx, ny, nz, steps = 48, 24, 12, 150
    ext = dict(geometry="duct") if faces is None else dict(geometry="duct", faces=faces)
    text = lbm.make_inputs(nx, ny, nz, obst1=(12.5, 11.5, 0.0), r1=4.0, re=40.0, umax=0.04, tmax=steps, les=les,
                           cs=0.02, model=model, **ext)
    with lbm.Solver(text) as s:
        s.step(steps)
        f, mask, om, F = s.populations(), s.mask(), s.params()["omega"], s.forces()
    assert (mask >= lbm.NODE["DIR_WEST"]).any()
    o = OracleRun(nx, ny, nz, mask, om, model=lbm.MODELS[model], les=les, cs=0.02, u_in=0.04, init_kind=0,
                  init_u=0.04)
    o.step(steps)
    err, drho = _compare(f, o.fa, mask)
    assert err < RTOL and drho < 1e-5, (err, drho)
    assert rel_l2(F[:, 0], np.array(o.forces)[: len(F), 0]) < FTOL


@pytest.mark.parametrize("prec,rel", [("fp16", 2.0 ** -11), ("bf16", 2.0 ** -8)])
@pytest.mark.parametrize("halfway", [0, 1])
def test_fp16_bf16_one_step_vs_oracle(product, prec, rel, halfway):
    """One FP16 / BF16 step from the stored populations of a developed
    channel flow matches the oracle's FP32 step from the same values to the
    storage rounding of the stored deviation f - feq(1, (UMAX, 0, 0)), the
    MRT model's own equilibrium: half an ulp of the format, doubled for
    margin.  A per-value check of the reduced-precision pull, the deviation
    collision and the conversions, sharper than the trajectory comparison
    against the FP64 twin"""
    lbm = product
    kw = dict(bounceback="halfway") if halfway else {}
    with lbm.Solver(_chan_inputs(lbm, 60, **kw)) as s:
        s.step(60)
        f_dev = s.populations()
    with lbm.Solver(_chan_inputs(lbm, 60, precision=prec, **kw)) as s:
        s.set_populations(f_dev)
        g0 = s.populations()
        s.step(1)
        g1, mask, om = s.populations(), s.mask(), s.params()["omega"]
        off = s.storage_offsets().astype(np.float64)[:, None, None, None]
    o = OracleRun(NX, NY, NZ, mask, om, model=0, les=1, cs=0.01, u_in=0.05, f0=g0, halfway=halfway)
    o.step(1)
    bound = 2 * rel * np.abs(o.fa - off) + 2e-7
    fl = np.broadcast_to(_fluid(mask), g1.shape)
    bad = (np.abs(g1 - o.fa) > bound) & fl
    assert not bad.any(), (int(bad.sum()), float(np.abs(g1 - o.fa)[fl].max()))
    # the bound resolves the step: without the update, or with the result one
    # node off in x, many values would fall outside it (oracle on the CPU:
    # 74 % / 85 % for FP16, 10 % / 40 % for BF16)
    n = fl.sum()
    assert ((np.abs(g0 - o.fa) > bound) & fl).sum() > 0.05 * n
    assert ((np.abs(np.roll(o.fa, 1, axis=-1) - o.fa) > bound) & fl).sum() > 0.3 * n


def test_lbm_run_command_writes_the_reference_outputs(product, tmp_path):
    """lbm_run, the reference programs' main() as a command: a run record in,
    the reference's timing line out, and the same output files as the
    handle writes after the same steps"""
    import subprocess

    from lbm_multigpu_gb300 import build

    lbm = product
    text = _chan_inputs(lbm, 30)
    (tmp_path / "case.inputs").write_text(text)
    exe = build.build_run()
    r = subprocess.run([str(exe), "case.inputs"], cwd=tmp_path, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    assert r.stdout.startswith("Time taken for main kernel: ") and r.stdout.rstrip().endswith("MLUPS)")
    ref = tmp_path / "api"
    ref.mkdir()
    with lbm.Solver(text) as s:
        s.step(30)
        s.write_outputs(str(ref / "case"))
    for name in ("case.inputs", "case_part0.dat", "case_slice.dat", "case.force"):
        assert (tmp_path / name).read_bytes() == (ref / name).read_bytes(), name
    bad = subprocess.run([str(exe), "missing.inputs"], cwd=tmp_path, capture_output=True, text=True, timeout=60)
    assert bad.returncode == 1 and "cannot read" in bad.stderr


def test_set_geometry_and_write_tecplot(product, tmp_path):
    """lbm_set_geometry: a caller's mask on the base level, NULL back to the
    record's analytic geometry; lbm_write_tecplot: the same tecplot files as
    lbm_write_outputs writes"""
    lbm = product
    with lbm.Solver(_chan_inputs(lbm, 10)) as s:
        m0 = s.mask()
        m1 = m0.copy()
        m1[:, 5:8, 40:44] = lbm.NODE["BODY"]
        s.set_geometry(m1)
        assert np.array_equal(s.mask(), m1)
        s.set_geometry(None)
        assert np.array_equal(s.mask(), m0)
        s.step(3)
        s.write_tecplot(str(tmp_path / "t"))
        s.write_outputs(str(tmp_path / "o"))
    for suffix in ("_part0.dat", "_slice.dat"):
        assert (tmp_path / f"t{suffix}").read_bytes() == (tmp_path / f"o{suffix}").read_bytes()
    assert not (tmp_path / "t.force").exists()


def _run_layout(lbm, text, steps, levels=1):
    with lbm.Solver(text) as s:
        s.step(steps)
        out = [s.populations(l) for l in range(levels)] + [s.forces(steps)]
        if "\nVELAV: \t1\n" in text:
            out.append(s.stats())
    return out


def test_ragged_width_channel_vs_oracle(product):
    """a width that is not a multiple of 32 (70: the last 32-node block of
    every row holds 26 padding lanes) in the default blocked layout, with
    half-way walls and inlet noise, against the oracle after 30 steps"""
    lbm = product
    steps, nx = 30, 70
    text = lbm.make_inputs(nx, 24, 6, obst1=(20.5, 11.5, 0.0), r1=4.0, re=60.0, umax=0.05, tmax=steps, les=1,
                           cs=0.01, geometry="channel_square", bounceback="halfway", inlet_noise=0.01, seed=9)
    with lbm.Solver(text) as s:
        s.step(steps)
        f, mask, om = s.populations(), s.mask(), s.params()["omega"]
    o = OracleRun(nx, 24, 6, mask, om, model=0, les=1, cs=0.01, u_in=0.05, init_u=0.05, noise_amp=0.01, seed=9,
                  halfway=1)
    o.step(steps)
    err, drho = _compare(f, o.fa, mask)
    assert err < RTOL and drho < 1e-5, (err, drho)


@pytest.mark.parametrize("precision", ["fp32", "fp16"])
def test_mapped_host_buffers_match_pageable(product, precision):
    """page-locked host buffers are read and written by the layout kernels
    directly (no staging copy): set from and get into pinned memory give
    the same values bit for bit as pageable numpy arrays, and the run that
    follows is the same"""
    torch = pytest.importorskip("torch")
    lbm = product
    text = lbm.make_inputs(96, 40, 12, obst1=(30.5, 19.5, 0.0), r1=4.0, re=60.0, umax=0.05, tmax=40, les=1, cs=0.01,
                           geometry="channel_square", precision=precision, inlet_noise=0.01, bounceback="halfway")
    with lbm.Solver(text) as s:
        s.step(7)
        f0 = s.populations()
        pinned_out = torch.empty(f0.shape, dtype=torch.float32, pin_memory=True).numpy()
        s.populations(out=pinned_out)
        np.testing.assert_array_equal(pinned_out, f0)
        g = f0.copy()
        g[:, :, 10:30, 20:60] *= np.float32(1.001)
        pinned_in = torch.empty(f0.shape, dtype=torch.float32, pin_memory=True).numpy()
        pinned_in[...] = g
        s.set_populations(pinned_in)
        a_set = s.populations()
        s.step(5)
        a_run = s.populations()
    with lbm.Solver(text) as s:
        s.step(7)
        s.set_populations(g)
        b_set = s.populations()
        s.step(5)
        b_run = s.populations()
    np.testing.assert_array_equal(a_set, b_set)
    np.testing.assert_array_equal(a_run, b_run)


@pytest.mark.parametrize("case", ["channel_fp32", "channel_fp16", "channel_bf16", "refine_fp16", "cavity_fp32",
                                  "duct_fp16"])
def test_population_layouts_are_bit_exact(product, case):
    """the blocked population layout (the 19 populations of 32 x-consecutive
    nodes together) runs the same arithmetic as the structure-of-arrays
    layout: identical populations, statistics and force histories after 40
    steps for half-way channels with inlet noise and statistics, a two-level
    refinement, the lid-driven cavity and a duct with alternate boundaries"""
    lbm = product
    steps = 40
    prec = case.split("_")[1]
    levels = 1
    if case.startswith("channel"):
        kw = dict(precision=prec, bounceback="halfway", inlet_noise=0.01, seed=5, velav=1, start_velav=10,
                  start_velfluc=25)
        make = lambda lay: _chan_inputs(lbm, steps, layout=lay, **kw)  # noqa: E731
    elif case.startswith("refine"):
        levels = 2
        make = lambda lay: lbm.make_inputs(  # noqa: E731
            128, 48, 8, obst1=(40.5, 23.5, 0.0), r1=3.0, re=60.0, umax=0.05, tmax=steps, les=1, cs=0.01,
            refinement=1, lr_dims=(48, 48, 16), lr_factor=0.5, lr_origin=(28.25, 12.25, -0.75),
            geometry="channel_square", cf_time="linear", precision=prec, layout=lay)
    elif case.startswith("cavity"):
        make = lambda lay: lbm.make_inputs(40, 40, 40, umax=0.05, tmax=steps, model="BGK", geometry="cavity",  # noqa
                                           tau=0.6, lid_velocity=(0.05, 0, 0), lid_face="+z", precision=prec,
                                           layout=lay)
    else:
        make = lambda lay: lbm.make_inputs(  # noqa: E731
            48, 24, 12, obst1=(12.5, 11.5, 0.0), r1=4.0, re=40.0, umax=0.04, tmax=steps, les=1, cs=0.02,
            model="MRT", geometry="duct", faces=("DIR_WEST", "NEU_EAST", "YSYM_BOT", "YSYM_TOP", "ZSYM_BOT",
                                                 "ZSYM_TOP"), precision=prec, layout=lay)
    a = _run_layout(lbm, make("soa"), steps, levels)
    assert np.isfinite(a[0]).all()
    for lay in ("blocked",):
        b = _run_layout(lbm, make(lay), steps, levels)
        for x, y in zip(a, b):
            np.testing.assert_array_equal(x, y)


def test_checkpoint_layout_must_match(product, tmp_path):
    """raw populations of a blocked-layout checkpoint are not read back into
    a structure-of-arrays handle"""
    lbm = product
    path = str(tmp_path / "blk.ckpt")
    with lbm.Solver(_chan_inputs(lbm, 10, precision="fp16", layout="blocked")) as s:
        s.step(5)
        s.save_state(path)
    with lbm.Solver(_chan_inputs(lbm, 10, precision="fp16", layout="soa")) as s:
        with pytest.raises(lbm.LbmError, match="layout"):
            s.restore_state(path)


def test_c2_benchmark_channel_vs_oracle(product):
    """the channel exactly as bench.py runs it (its own record: 512x128x128,
    MRT + Smagorinsky CS = 0.01, tau0 = 0.52, square body of side 16 at
    x = 128 with half-way bounce-back, 1 % seeded inlet noise, zero-gradient
    outlet, periodic z) against the oracle at full size after 60 steps:
    velocity relative L2 and density within 1e-5, drag within 1e-4"""
    import bench

    lbm = product
    steps = 60
    with lbm.Solver(bench.inputs_text("fp32", steps)) as s:
        s.step(steps)
        f, mask, om, F = s.populations(), s.mask(), s.params()["omega"], s.forces()
    o = OracleRun(bench.NX, bench.NY, bench.NZ, mask, om, model=0, les=1, cs=0.01, u_in=0.05, init_u=0.05,
                  noise_amp=0.01, seed=12345, halfway=1)
    o.step(steps)
    err, drho = _compare(f, o.fa, mask)
    assert err < RTOL and drho < 1e-5, (err, drho)
    Fo = np.array(o.forces)[: len(F)]
    assert rel_l2(F[:, 0], Fo[:, 0]) < FTOL
    assert np.abs(F[:, 1] - Fo[:, 1]).max() < FTOL * np.abs(Fo[:, 0]).max()
    # the flow developed past the body: the wake differs from the inlet state
    _, j = moments(f)
    assert np.abs(j[0][:, 40:90, 140:200] - 0.05).max() > 1e-3


def test_c3_configured_patch_vs_oracle(product):
    """the two-level refinement as bench.py runs it: coarse 256x128x64
    channel with a circular cylinder of diameter 12, the configured 96x64x64
    fine patch bounded in z, linear temporal interpolation, 1 % noise;
    10 coarse steps (20 fine) against the oracle on both levels"""
    import bench

    lbm = product
    steps = 10
    with lbm.Solver(bench.c3_inputs(steps)) as s:
        s.step(steps)
        fc, ff, mc, mf, pr = s.populations(0), s.populations(1), s.mask(0), s.mask(1), s.params()
    fx, fy, fz = bench.C3_PATCH["lr_dims"]
    x0, y0, z0 = bench.C3_PATCH["lr_origin"]
    r = Refine(cnx=256, cny=128, cnz=64, fnx=fx, fny=fy, fnz=fz, lrx0=x0, lry0=y0, lrz0=z0, lrfactor=0.5,
               lrlevel=2, order=2, cs=0.01, omega_c=pr["omega"], omega_f=pr["omega_lr"], quirk_fc_top_zflip=1,
               zbounded=1, cz0=int(z0))
    o = OracleRun(256, 128, 64, mc, pr["omega"], les=1, cs=0.01, noise_amp=0.01, seed=12345,
                  refine=dict(r=r, mask=mf, omega_f=pr["omega_lr"]), cf_time=True)
    o.step(steps)
    assert _compare(fc, o.fa, mc)[0] < RTOL
    _, jf = moments(ff)
    _, jo = moments(o.ffa)
    assert rel_l2(jf[:, mf != 2], jo[:, mf != 2]) < RTOL


@pytest.mark.parametrize("nx,ny,nz", [(31, 13, 5), (33, 12, 6), (64, 12, 5), (70, 24, 6)])
def test_statistics_readback(product, nx, ny, nz):
    """the statistics without their row padding, into pageable and into pinned
    memory: after one step from start_velav 0 the mean is the momentum of the
    populations (19 FP32 terms below 1/3 each: 19 x 2^-24 at most apart), and
    nothing is written at solid nodes"""
    torch = pytest.importorskip("torch")
    lbm = product
    text = lbm.make_inputs(nx, ny, nz, obst1=(8.5, 5.5, 0.0), r1=2.0, re=60.0, umax=0.05, tmax=10, les=1, cs=0.01,
                           geometry="channel_square", velav=1, start_velav=0, start_velfluc=5)
    with lbm.Solver(text) as s:
        s.step(1)
        st, f, mask = s.stats(), s.populations().astype(np.float64), s.mask()
        pin = torch.empty((4, nz, ny, nx), dtype=torch.float32, pin_memory=True)
        lbm._check(s._lib.lbm_get_stats(s._h, 0, pin.data_ptr()))
    np.testing.assert_array_equal(st, pin.numpy())
    solid = np.isin(mask, [lbm.NODE["WALL"], lbm.NODE["BODY"]])
    for k, c in enumerate((CX, CY)):
        np.testing.assert_allclose(st[k][~solid], np.tensordot(c, f, 1)[~solid], rtol=0, atol=19 * 2.0 ** -24)
    assert not st[:, solid].any() and not st[2:].any()


def test_step_graphs_grow_after_a_short_call(product):
    """a short call leaves graphs of 2, 4 and 8 steps; a long one after it
    grows to batches of 16: beside two kernels a step, at most one launch per
    batch of 16 and one for each of the shorter ones and the counter's start"""
    lbm = product
    with lbm.Solver(lbm.make_inputs(64, 24, 12, obst1=(18.5, 11.5, 0.0), r1=4.0, re=60.0, umax=0.05, tmax=1000, les=1,
                                    cs=0.01, bounceback="halfway")) as s:
        s.step(20)
        n0 = s.launch_count()
        s.step(640)
        assert s.launch_count() - n0 <= 2 * 640 + 640 // 16 + 12
