"""Split products on host operands whose schedule divides tiles' reductions (stream-K), in the call over
all of C, in the pipelined path's column blocks, or in both: the bits of the call on device
pointers, as for every other size (tests/test_gpu_host_pipeline.py)."""
import pytest

from mojoblas_b200 import _lib as L
from tests.gpu_util import need_gpu

pytestmark = pytest.mark.gpu

# m n k >= 2^34 and n >= 4096 (the pipelined path).  128 x 256 tiles on 148 SMs, whole call / block of columns:
# 320 / 40, 2048 / 256, 1344 / 192, and 320 with a ragged edge on every side
SHAPES = [(2560, 4096, 1700), (8192, 8192, 260), (8192, 5376, 400), (2500, 4100, 1731)]


@pytest.mark.parametrize("mode", [L.MODE_BF16X3, L.MODE_BF16X6], ids=["bf16x3", "bf16x6"])
@pytest.mark.parametrize("ta,tb", [("N", "N"), ("T", "T")])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_host_call_matches_device_call(mode, ta, tb, m, n, k):
    torch = need_gpu()
    lib = L.load()
    g = torch.Generator(device="cuda")
    g.manual_seed(m + n + k)

    def uniform(rows, cols):  # column-major rows x cols
        return torch.rand((cols, rows), generator=g, device="cuda") * 2 - 1

    a, b = uniform(*((m, k) if ta == "N" else (k, m))), uniform(*((k, n) if tb == "N" else (n, k)))
    lda, ldb = a.shape[1], b.shape[1]
    c = torch.full((n, m), 7.0, device="cuda")
    hc = torch.full((n, m), 7.0).pin_memory()
    ha, hb = a.cpu().pin_memory(), b.cpu().pin_memory()
    torch.cuda.synchronize()
    for pa, pb, pc in ((a, b, c), (ha, hb, hc)):
        assert lib.mbg_sgemm_ex(mode, ta.encode(), tb.encode(), m, n, k, 1.25, pa.data_ptr(), lda, pb.data_ptr(), ldb,
                                0.0, pc.data_ptr(), m) == 0, L.last_error()
        torch.cuda.synchronize()
    assert torch.equal(c.cpu().view(torch.int32), hc.view(torch.int32))
