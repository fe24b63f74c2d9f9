"""Column blocks of the pipelined host path take tiles of their own size, but divide a reduction as the call over
all of C does: the same bits as the call on device pointers, where the whole product shares tiles
among CTAs and where it does not (tests/test_gpu_host_pipeline.py has one size for every mode)."""
import pytest

from mojoblas_b200 import _lib as L
from tests.gpu_util import need_gpu

pytestmark = pytest.mark.gpu

CASES = [("f32", L.MODE_PLAIN, 4096, 4096, 1024),  # 128-tiles in the whole call, 64-tiles in its blocks
         ("f32", L.MODE_PLAIN, 256, 4096, 16401),  # 128-tiles shared by two CTAs; 64-tiles, parts of whole pairs of slabs
         ("f32", L.MODE_PLAIN, 130, 5003, 26800),  # by more, ragged
         ("f32", L.MODE_PLAIN, 63, 4100, 66600),   # 64-tiles shared in both
         ("f64", L.MODE_PLAIN, 4096, 4096, 1030),  # 128-tiles in the whole call, 64-tiles in its blocks
         ("f64", L.MODE_PLAIN, 128, 4100, 32800),  # shared 64-tiles
         ("f32", L.MODE_BF16X6, 4096, 4096, 1100), ("f32", L.MODE_BF16X6, 250, 4100, 16900),
         ("f32", L.MODE_BF16X3, 250, 4100, 16900)]


@pytest.mark.parametrize("ta,tb", [("N", "T"), ("T", "N")])
@pytest.mark.parametrize("beta", [0.0, 0.5])
@pytest.mark.parametrize("dt,mode,m,n,k", CASES)
def test_blocks_match_device_call(dt, mode, m, n, k, ta, tb, beta):
    torch = need_gpu()
    lib = L.load()
    dtype = torch.float32 if dt == "f32" else torch.float64
    g = torch.Generator(device="cuda")
    g.manual_seed(m + n + k)

    def uniform(rows, cols):  # column-major rows x cols
        return torch.rand((cols, rows), generator=g, device="cuda", dtype=dtype) * 2 - 1

    a, b = uniform(*((m, k) if ta == "N" else (k, m))), uniform(*((k, n) if tb == "N" else (n, k)))
    lda, ldb = a.shape[1], b.shape[1]
    c = uniform(m, n)
    hc, ha, hb = c.cpu().pin_memory(), a.cpu().pin_memory(), b.cpu().pin_memory()
    torch.cuda.synchronize()
    for pa, pb, pc in ((a, b, c), (ha, hb, hc)):
        args = (ta.encode(), tb.encode(), m, n, k, 1.25, pa.data_ptr(), lda, pb.data_ptr(), ldb, beta, pc.data_ptr(), m)
        st = lib.mbg_sgemm_ex(mode, *args) if dt == "f32" else lib.mbg_dgemm_ex(mode, 0, *args)
        assert st == 0, L.last_error()
        torch.cuda.synchronize()
    word = torch.int32 if dt == "f32" else torch.int64
    assert torch.equal(c.cpu().view(word), hc.view(word))
