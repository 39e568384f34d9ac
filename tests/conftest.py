"""pytest configuration: the `gpu` marker and session fixtures that build the
product library, the oracle and the test-only host build of the product's
per-cell operators."""
from __future__ import annotations

import ctypes
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
for p in (ROOT, ROOT / "tests", ROOT / "oracle"):
    if str(p) not in sys.path:
        sys.path.insert(0, str(p))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (GB300, sm_103a)")
    # the tests' temporary files stay inside the working tree (git-ignored)
    if not config.option.basetemp:
        config.option.basetemp = str(ROOT / ".pytest_tmp")


@pytest.fixture(scope="session")
def product():
    """the product package with its CUDA library built in-tree"""
    from lbm_multigpu_gb300 import build

    build.build()
    import lbm_multigpu_gb300 as lbm

    lbm.library()
    return lbm


@pytest.fixture(scope="session")
def orc():
    from oracle_bindings import oracle

    return oracle()


@pytest.fixture(scope="session")
def cellops(tmp_path_factory):
    """host build of lbm_multigpu_gb300/csrc/d3q19.cuh (test-only shim)"""
    from lbm_multigpu_gb300.build import nvcc

    out = tmp_path_factory.mktemp("cellops") / "cellops.so"
    src = ROOT / "tests" / "native" / "cell_ops_shim.cu"
    r = subprocess.run([nvcc(), "-O2", "-std=c++17", "-Xcompiler", "-fPIC,-ffp-contract=off", "-shared", "-o",
                        str(out), str(src)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = ctypes.CDLL(str(out))
    lib.cell_philox_uniform.restype = ctypes.c_float
    return lib


@pytest.fixture(scope="session")
def fakecuda(tmp_path_factory):
    """the library's host sources over a stand-in for the CUDA runtime and the
    kernels (test-only, tests/native/fake_cuda.cpp): bookkeeping and error
    paths without a GPU"""
    from lbm_multigpu_gb300.build import CSRC, nvcc

    d = tmp_path_factory.mktemp("fakecuda")
    inc = "-I" + str(Path(nvcc()).resolve().parents[1] / "include")
    cxx = ["g++", "-O1", "-std=c++17", "-fPIC", inc]
    srcs = [CSRC / "lbm_host.cpp", CSRC / "lbm_sgs.cpp", CSRC / "lbm_ensemble.cpp", ROOT / "tests" / "native" / "fake_cuda.cpp"]
    objs = [str(d / (p.stem + ".o")) for p in srcs]
    for p, r in [(p, subprocess.Popen([*cxx, "-c", str(p), "-o", o])) for p, o in zip(srcs, objs)]:
        assert r.wait() == 0, p
    names = {f: {line.split()[-1] for line in subprocess.run(["nm", *f, *objs], capture_output=True, text=True,
                                                            check=True).stdout.splitlines() if len(line.split()) > 1}
             for f in (("-u",), ("--defined-only",))}
    rest = sorted(n for n in names["-u",] - names["--defined-only",] if n.startswith(("cuda", "_ZN3lbm")))
    stubs = d / "stubs.c"
    stubs.write_text("".join(f"long {n}(void) {{ return 0; }}\n" for n in rest))
    out = d / "fakecuda.so"
    r = subprocess.run(["gcc", "-O1", "-fPIC", "-c", str(stubs), "-o", str(d / "stubs.o")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run(["g++", "-shared", "-o", str(out), *objs, str(d / "stubs.o")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = ctypes.CDLL(str(out))
    lib.fake_calls.restype = lib.fake_trace.restype = ctypes.c_long
    lib.lbm_last_error.restype = ctypes.c_char_p
    return lib


@pytest.fixture(scope="session")
def golden():
    import numpy as np

    import json

    g = ROOT / "tests" / "golden"
    runs, meta = {}, {}
    for stem in ("runs", "runs_1k"):  # the 1000-step channel is its own file
        runs.update(dict(np.load(g / f"{stem}.npz")))
        meta.update(json.loads((g / f"{stem}.json").read_text()))
    return dict(cells=np.load(g / "cells.npz"), runs=runs, meta=meta, dir=g)
