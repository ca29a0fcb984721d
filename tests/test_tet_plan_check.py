"""How many contributor words the gradient pass stages per cluster (tc_dent of the tet plan) is part of the plan's
invariant checks: too few would leave diagonal items without theirs, too many overrun the pass's shared memory, and
the copies move eight at a time."""

import ctypes
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from litepgo_b200 import mesh


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no host C++ compiler")
    csrc = ROOT / "litepgo_b200" / "csrc"
    out = tmp_path_factory.mktemp("plancheck") / "libplancheck.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", str(csrc), "-I", "/usr/local/cuda/include",
                    str(ROOT / "tests" / "tet_plan_check_host.cpp"), str(csrc / "lpg_plan.cpp"), "-o", str(out)],
                   check=True)
    lib = ctypes.CDLL(str(out))
    lib.check_plan.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.POINTER(ctypes.c_int32)] + [ctypes.c_int] * 3
    return lambda X, tets, cluster=0, add=0, drop=0: lib.check_plan(
        X.shape[0], tets.shape[0], np.ascontiguousarray(tets, np.int32).ctypes.data_as(ctypes.POINTER(ctypes.c_int32)),
        cluster, add, drop)


@pytest.mark.parametrize("box", [1, 3, 9])
def test_staged_contributors(check, box):
    X, tets = mesh.make_box(box)
    assert check(X, tets) == 0
    for cluster in (0, -1):
        for add in (-1, 1, -8, 8, 1 << 12):
            assert check(X, tets, cluster, add) == -1, (cluster, add)
    assert check(X, tets, drop=1) == -1
