"""Batches of steps (direct steps, CUDA graphs of 4, 8 and 16, in the order
that calls of any length meet them) equal single steps bit for bit, in the
formats and record options that test_gpu_parity's batches do not have."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CALLS = [2, 2, 2, 4, 4, 4, 8, 8, 12, 12, 20, 20, 3, 64, 17, 96]
WEIGHTS = "data/sgs_mlp.bin"


def _kind(lbm, kind):
    kw = dict(obst1=(18.5, 11.5, 0.0), r1=4.0, re=60.0, umax=0.05, tmax=400, les=1, cs=0.01, inlet_noise=0.01, seed=5)
    if kind.startswith("refined"):
        kw.update(refinement=1, lr_dims=(32, 32, 12), lr_factor=0.5, lr_origin=(12.25, 4.25, 2.25), cf_time="linear",
                  precision=kind.split("_")[1])
    elif kind.startswith("closure"):      # no body: launches may begin early behind an evaluation of the closure
        _, every, precision = kind.split("_")
        kw.update(geometry="channel", bounceback="halfway", sgs="mlp", sgs_every=int(every), precision=precision,
                  sgs_weights=str(lbm.LIB_PATH.parent.parent / WEIGHTS))
    elif kind == "cavity":
        kw = dict(re=100.0, umax=0.05, tmax=400, les=0, model="BGK", geometry="cavity", lid_velocity=(0.05, 0.0, 0.0),
                  lid_face="+z")
    return lbm.make_inputs(64, 24, 12, **kw)


@pytest.mark.parametrize("kind", ["refined_fp32", "refined_fp16", "refined_bf16", "refined_fp64", "closure_1_fp32",
                                  "closure_4_fp32", "closure_6_fp16", "cavity", "body"])
def test_batches_equal_single_steps(product, kind):
    lbm = product
    text, res = _kind(lbm, kind), []
    for calls in (CALLS, [1] * sum(CALLS)):
        with lbm.Solver(text) as s:
            for n in calls:
                s.step(n)
            res.append([s.populations(k) for k in range(s.nlevels)] + [s.forces()])
    assert np.isfinite(res[0][0]).all()
    for a, b in zip(*res):
        np.testing.assert_array_equal(a, b)


def test_closure_steps_of_several_threads(product):
    """handles with the closure, each of its own thread, and an ensemble with
    it, all capturing graphs: every one has the result of a thread alone"""
    import threading

    lbm = product
    text, weights = _kind(lbm, "closure_1_fp32"), np.fromfile(lbm.LIB_PATH.parent.parent / WEIGHTS, np.float32)

    def flow():
        with lbm.Solver(text) as s:
            for n in (16, 16, 16, 40):
                s.step(n)
            return s.populations()

    def boxes():
        with lbm.Ensemble([32, 16], 0.55, sgs="mlp") as e:
            e.set_mlp(weights)
            e.init_turbulence(3)
            e.step(40)
            return e.populations(0)

    want, wrong = {f: f() for f in (flow, boxes)}, []

    def work(f):
        for _ in range(12):
            try:
                np.testing.assert_array_equal(f(), want[f])
            except Exception as e:   # an error code, or another result
                wrong.append(str(e)[:200])

    threads = [threading.Thread(target=work, args=(f,)) for f in (flow, flow, flow, boxes)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
