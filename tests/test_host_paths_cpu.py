"""The library's host code over a stand-in for the CUDA runtime
(tests/native/fake_cuda.cpp): index arithmetic at sizes that no test machine
holds, and what is left behind when a call of the runtime fails."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest


def _ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


@pytest.fixture
def fake(fakecuda):
    fakecuda.fake_reset()
    yield fakecuda
    fakecuda.fake_reset()


def _train(fake, n, batch, steps, seed=9):
    """the (start, size) of every mini-batch of lbm_mlp_train"""
    P = np.zeros(fake.lbm_mlp_param_count(), np.float32)
    x = ctypes.c_void_p(16)   # never read: the kernels are stand-ins
    rc = fake.lbm_mlp_train(x, x, n, batch, steps, ctypes.c_float(1e-3), seed, _ptr(P), None, None)
    assert rc == 0, fake.lbm_last_error()
    out = (ctypes.c_longlong * (2 * steps))()
    assert fake.fake_trace(out, 2 * steps) == 2 * steps
    return [(out[2 * i], out[2 * i + 1]) for i in range(steps)]


@pytest.mark.parametrize("n,batch", [(1 << 30, 1 << 30), (1_200_000_000, 1_000_000_000), (2 ** 31 - 1, 2 ** 30)])
def test_batches_stay_inside_the_samples(fake, n, batch):
    """batches near 2^31 samples (position + batch passes the range of an
    int): each lies within the permutation"""
    for start, size in _train(fake, n, batch, 4):
        assert 0 <= start and start + size <= n
