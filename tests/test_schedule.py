"""The schedules' arithmetic (mojoblas_b200/csrc/schedule.cuh, plain C++) compiled by the host
compiler and checked at sizes that no test can run on the device."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
SOURCE = r'''
#include "mojoblas_b200/csrc/schedule.cuh"
using namespace mbg;
extern "C" {
i64 slab_count(i64 k, int depth) { return k_slabs(k, depth).n; }
int slab_left(i64 k, int depth, i64 kb) {
    const KSlabs s = k_slabs(k, depth);
    return k_left(int(s.n), s.last, int(kb), depth);
}
}
'''


@pytest.fixture(scope="module")
def sched(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("schedule")
    (d / "check.cpp").write_text(SOURCE)
    subprocess.run([cxx, "-std=c++17", "-O2", "-fPIC", "-shared", "-fwrapv", "-I", str(ROOT), str(d / "check.cpp"), "-o",
                    str(d / "check.so")], check=True)
    lib = C.CDLL(str(d / "check.so"))
    lib.slab_count.restype = C.c_int64
    lib.slab_count.argtypes = [C.c_int64, C.c_int]
    lib.slab_left.argtypes = [C.c_int64, C.c_int, C.c_int64]
    return lib


@pytest.mark.parametrize("k", [0, 1, 31, 32, 33, 64, 2**31 - 33, 2**31 - 32, 2**31 - 31, 2**31 - 1, 2**31, 2**31 + 1, 2**35 + 7])
def test_last_slab_ends_with_the_reduction(sched, k):
    """No slab reaches past k, also where the slab's end passes 2^31."""
    n = sched.slab_count(k, 32)
    assert n == -(-k // 32)
    for kb in {0, 1, n // 2, n - 2, n - 1}:
        if 0 <= kb < n:
            assert sched.slab_left(k, 32, kb) == min(32, k - 32 * kb), kb
