"""Grouped split sgemm gives the same bits whatever the operands' alignment: pairs of k that are 8-byte aligned in every
row are loaded together, others one by one, with the same arithmetic.  Shapes at the edges of row groups,
tiles and k slabs, and enough of them that slabs are prefetched across tiles."""
import pytest

from mojoblas_b200 import _lib as L
from tests.gpu_util import need_gpu

pytestmark = pytest.mark.gpu
SHAPES = [(m, n, k) for m in (1, 32, 33, 128, 130) for n in (1, 64, 129) for k in (1, 2, 31, 32, 33, 64, 96, 130)] * 4


@pytest.mark.parametrize("mode", [L.MODE_BF16X3, L.MODE_BF16X6], ids=["bf16x3", "bf16x6"])
@pytest.mark.parametrize("ta,tb", [("T", "N"), ("T", "T"), ("N", "N"), ("N", "T")])
def test_layouts_agree(mode, ta, tb):
    torch = need_gpu()
    lib = L.load()
    g = torch.Generator(device="cuda")
    g.manual_seed(11)
    values = [(torch.rand((k, m) if ta == "N" else (m, k), generator=g, device="cuda") * 2 - 1,
               torch.rand((n, k) if tb == "N" else (k, n), generator=g, device="cuda") * 2 - 1) for m, n, k in SHAPES]

    def place(t, pad, off):  # the matrix with a leading dimension `pad` longer, `off` floats into its buffer
        buf = torch.full((off + t.shape[0] * (t.shape[1] + pad),), float("nan"), device="cuda")
        buf[off:].view(t.shape[0], -1)[:, :t.shape[1]] = t
        return buf

    results = []
    for pad, off in ((0, 0), (1, 0), (0, 1), (2, 2), (4, 0)):
        probs, held = (L.SgemmProblem * len(SHAPES))(), []
        for i, (m, n, k) in enumerate(SHAPES):
            a, b = (place(t, pad, off) for t in values[i])
            c = torch.full((n, m), 9.0, device="cuda")
            held.append((a, b, c))
            probs[i] = L.SgemmProblem(ta.encode(), tb.encode(), m, n, k, 1.5, 0.0, a.data_ptr() + 4 * off,
                                      values[i][0].shape[1] + pad, b.data_ptr() + 4 * off, values[i][1].shape[1] + pad,
                                      c.data_ptr(), m)
        torch.cuda.synchronize()
        assert lib.mbg_sgemm_grouped(mode, len(SHAPES), probs) == 0, L.last_error()
        torch.cuda.synchronize()
        results.append([c for _, _, c in held])
    for other in results[1:]:
        for shape, x, y in zip(SHAPES, results[0], other):
            assert torch.equal(x, y), shape
