"""The FP64 square root and reciprocal of the device code (Newton's iteration
from FP32 approximations), and the FP64 collision that uses them, against
IEEE arithmetic on the host."""
from __future__ import annotations

import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

from oracle_bindings import CX, CY, CZ, W

pytestmark = pytest.mark.gpu


def _ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


@pytest.fixture(scope="module")
def devops(tmp_path_factory):
    from lbm_multigpu_gb300.build import ARCH, NVCC_FLAGS, nvcc

    out = tmp_path_factory.mktemp("devops") / "devops.so"
    r = subprocess.run([nvcc(), *ARCH, *NVCC_FLAGS, "-shared", "-o", str(out),
                        str(Path(__file__).parent / "native" / "device_ops_shim.cu")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(str(out))


def _map(devops, what, x):
    y = np.empty_like(x)
    assert devops.dev_map(what, _ptr(x), _ptr(y), len(x)) == 0
    return y


def _arguments():
    """positive: even in the logarithm over all of FP64 and over the FP32
    path's range, the latter's ends, all-ones and all-zero mantissas"""
    rng = np.random.default_rng(5)
    m = 1 + rng.random(200_000)
    wide = np.ldexp(m, rng.integers(-1022, 1023, len(m)))
    inside = np.ldexp(m, rng.integers(-100, 100, len(m)))
    ends = [np.nextafter(v, t) for v in (2.0 ** -100, 2.0 ** 100) for t in (0, v, np.inf)]
    e = np.arange(-1022, 1024)
    return np.concatenate([wide, inside, ends, np.ldexp(1.0, e), np.ldexp(np.nextafter(2.0, 1), e[:-1]),
                           np.ldexp(1 + 2.0 ** -23, e), np.ldexp(1 + 2.0 ** -23 - 2.0 ** -52, e)])


@pytest.mark.parametrize("what", ["lsqrt", "dsqrt", "lrcp"])
def test_newton_square_root_and_reciprocal(devops, what):
    """within an ulp of the correctly rounded result, and equal to it but for
    near ties: with the seed's relative error d below 2^-21 the last step's
    argument is off by 1.5 d^3 (square root; d^4 in the reciprocal), under
    2^-10 of an ulp, before its one rounding.  Outside the FP32 range, and at
    0, subnormals, infinity, NaN and negative values, IEEE's results."""
    code = ["lsqrt", "dsqrt", "lrcp"].index(what)
    ref = (lambda v: 1.0 / v) if what == "lrcp" else np.sqrt
    x = _arguments()
    with np.errstate(all="ignore"):
        want, got = ref(x), _map(devops, code, x)
        fin = np.isfinite(want)
        ulps = np.abs(got - want)[fin] / np.spacing(want[fin])
        assert ulps.max() <= 1
        assert np.count_nonzero(ulps) <= 2.0 ** -7 * len(x)
        inside = (x >= 2.0 ** -100) & (x < 2.0 ** 100)
        np.testing.assert_array_equal(got[~inside], want[~inside])
        odd = np.array([0.0, -0.0, 5e-324, 2.2e-308, 1e-310, np.inf, -np.inf, np.nan, -1.0, -2.0 ** -50, -2.0 ** 120,
                        -5e-324])
        np.testing.assert_array_equal(_map(devops, code, odd), ref(odd))


@pytest.mark.parametrize("les", [0, 1])
def test_fp64_collision_on_the_device(devops, cellops, les):
    """collide_mrt_pop<double> on the device against the host build (sqrt and
    division): some 120 operations on values below 1/2, each rounded by at
    most 2^-54, give 7e-15"""
    rng = np.random.default_rng(17 + les)
    u = rng.uniform(-0.08, 0.08, (4000, 3))
    cu = u @ np.array([CX, CY, CZ], np.float64)
    rho = 1 + rng.uniform(-0.02, 0.02, (4000, 1))
    f = W * (rho + 3 * cu + 4.5 * cu ** 2 - 1.5 * (u ** 2).sum(1, keepdims=True))
    f = np.ascontiguousarray(f + 0.01 * W * rng.standard_normal(f.shape))
    om, cs = ctypes.c_double(1 / 0.52), ctypes.c_double(0.01)
    got, want = np.empty_like(f), f.copy()
    assert devops.dev_collide(les, om, cs, _ptr(f), _ptr(got), len(f)) == 0
    zero = ctypes.c_double(0.0)
    cellops.cell_collide_mrt_pop_d(0, 0, les, om, cs, zero, zero, _ptr(want), len(f))
    np.testing.assert_allclose(got, want, rtol=0, atol=7e-15)
