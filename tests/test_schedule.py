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
// The schedule of tiles_m x tiles_n tiles of nkb slabs on up to `sms` workers; returns the workers.
i64 plan(int tiles_m, int tiles_n, int nkb, i64 sms, i64* out) {
    i64 G = sms;
    const SkWork W = sk_plan(i64(tiles_m) * tiles_n, nkb, 0, 0, G, true);
    out[0] = W.dp_tiles; out[1] = W.sk_begin; out[2] = W.total;
    return G;
}
i64 range_begin(i64 begin, i64 total, i64 w, i64 workers) {
    SkWork W{};
    W.sk_begin = begin; W.total = total;
    return sk_range_begin(W, w, workers);
}
void place(int tiles_m, int tiles_n, int group, int t, int* tm, int* tn) {
    const TileAt at = tile_at(TileGrid{tiles_m, tiles_n, group}, t);
    *tm = at.tm; *tn = at.tn;
}
i64 kept(int tri, i64 tiles_m, i64 n, int bm, int bn) { return kept_tiles(tri, tiles_m, n, bm, bn); }
// The cut of tile t of the column block of `cols` tile columns from tn0 on.
int block_cut(int tiles_m, int tiles_n, int group, int nkb, i64 sms, int tn0, int cols, int t) {
    SkBlock B{};
    i64 G = sms;
    B.W = sk_plan(i64(tiles_m) * tiles_n, nkb, 0, 0, G, true);
    B.workers = G;
    B.whole = TileGrid{tiles_m, tiles_n, group};
    B.block = TileGrid{tiles_m, cols, group};
    B.tn0 = tn0;
    return sk_block_cut(B, t);
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
    lib.kept.restype = C.c_int64
    lib.kept.argtypes = [C.c_int, C.c_int64, C.c_int64, C.c_int, C.c_int]
    lib.plan.restype = lib.range_begin.restype = C.c_int64
    lib.plan.argtypes = [C.c_int, C.c_int, C.c_int, C.c_int64, C.POINTER(C.c_int64)]
    lib.range_begin.argtypes = [C.c_int64] * 4
    lib.block_cut.argtypes = [C.c_int] * 4 + [C.c_int64] + [C.c_int] * 3
    return lib


@pytest.mark.parametrize("k", [0, 1, 31, 32, 33, 64, 2**31 - 33, 2**31 - 32, 2**31 - 31, 2**31 - 1, 2**31, 2**31 + 1, 2**35 + 7])
def test_last_slab_ends_with_the_reduction(sched, k):
    """No slab reaches past k, also where the slab's end passes 2^31."""
    n = sched.slab_count(k, 32)
    assert n == -(-k // 32)
    for kb in {0, 1, n // 2, n - 2, n - 1}:
        if 0 <= kb < n:
            assert sched.slab_left(k, 32, kb) == min(32, k - 32 * kb), kb


@pytest.mark.parametrize("tiles_m,tiles_n,nkb,sms", [(20, 16, 54, 148), (64, 21, 13, 148), (17, 9, 1, 148), (33, 25, 7, 148),
                                                     (3, 50, 100, 148), (150, 1, 9, 148), (16, 16, 5, 100), (64, 32, 9, 148)])
def test_column_blocks_cut_tiles_as_the_whole_schedule(sched, tiles_m, tiles_n, nkb, sms):
    """Every tile of the whole product is in exactly one tile of the column blocks, cut at the slab where a
    worker's range of the whole schedule ends inside it, or not at all."""
    out = (C.c_int64 * 3)()
    workers = sched.plan(tiles_m, tiles_n, nkb, sms, out)
    dp, begin, total = out
    group = 16
    want = {}
    for t in range(tiles_m * tiles_n):
        tm, tn = C.c_int(), C.c_int()
        sched.place(tiles_m, tiles_n, group, t, C.byref(tm), C.byref(tn))
        assert (tm.value, tn.value) not in want
        want[tm.value, tn.value] = 0
        if total > begin and t >= dp:
            edges = {sched.range_begin(begin, total, w, workers) for w in range(workers + 1)}
            inside = [e - t * nkb for e in edges if t * nkb < e < (t + 1) * nkb]
            assert len(inside) <= 1  # no tile gets more than two partial sums
            want[tm.value, tn.value] = inside[0] if inside else 0
    got, tn0 = {}, 0
    while tn0 < tiles_n:
        cols = min(max(1, (tiles_n - tn0) // 3), tiles_n - tn0)
        for t in range(tiles_m * cols):
            tm, tn = C.c_int(), C.c_int()
            sched.place(tiles_m, cols, group, t, C.byref(tm), C.byref(tn))
            assert (tm.value, tn0 + tn.value) not in got
            got[tm.value, tn0 + tn.value] = sched.block_cut(tiles_m, tiles_n, group, nkb, sms, tn0, cols, t)
        tn0 += cols
    assert got == want


@pytest.mark.parametrize("bn", [64, 128, 256])
@pytest.mark.parametrize("tri", [0, 1, 2])
def test_tiles_that_a_mask_keeps(sched, tri, bn):
    for m, n in ((1, 1), (128, 128), (129, 130), (700, 700), (1025, 513), (513, 1025), (3000, 3000), (4096, 100)):
        tiles_m = -(-m // 128)
        want = sum(not (tri == 1 and 128 * tm + 128 <= bn * tn or tri == 2 and 128 * tm > bn * tn + bn - 1)
                   for tm in range(tiles_m) for tn in range(-(-n // bn)))
        assert sched.kept(tri, tiles_m, n, 128, bn) == want, (m, n)


def test_counting_kept_tiles_is_quick(sched):
    """On the launch path of every masked product: 65536 x 65536 has half a million tiles of 128 x 64."""
    import time
    best = float("inf")
    for _ in range(5):
        start = time.perf_counter()
        for bn in (64, 128, 256):
            sched.kept(1, 512, 65536, 128, bn)
        best = min(best, time.perf_counter() - start)
    assert best < 1e-4
