"""Split products whose reduction is shared by the CTAs of a cluster (few output tiles): edges of
tiles and of the slabs' division, every beta form, the triangle mask, and repeat calls with
the same bits.  Tolerances: those of tests/test_gpu_tc.py for the mode, against float64."""
import pytest

import mojoblas_b200 as mb
from tests.gpu_util import need_gpu
from tests.test_gpu_tc import tol_mode

pytestmark = pytest.mark.gpu
MODES = pytest.mark.parametrize("mode", [mb.BF16X3, mb.BF16X6], ids=["bf16x3", "bf16x6"])


@MODES
@pytest.mark.parametrize("ta,tb", [("N", "T"), ("T", "N")])
@pytest.mark.parametrize("beta", [0.0, 1.0, 0.5])
@pytest.mark.parametrize("m,n,k", [(1, 1, 4096), (129, 257, 33), (128, 256, 96), (500, 300, 2049), (1531, 1023, 2047),
                                   (512, 512, 512), (130, 1300, 8200), (2047, 1025, 300)])
def test_split_gemm_few_tiles(mode, ta, tb, beta, m, n, k):
    torch = need_gpu()
    g = torch.Generator(device="cuda")
    g.manual_seed(m + n + k)

    def uniform(*shape):
        return torch.rand(shape, generator=g, device="cuda") * 2 - 1

    lda, ldb, ldc = (m if ta == "N" else k) + 3, (k if tb == "N" else n) + 2, m + 5
    a, b, c0 = uniform(k if ta == "N" else m, lda), uniform(n if tb == "N" else k, ldb), uniform(n, ldc)
    av = a[:, :lda - 3].double()
    bv = b[:, :ldb - 2].double()
    ref = -1.25 * (av.T if ta == "N" else av) @ (bv.T if tb == "N" else bv) + beta * c0[:, :m].double().T
    outs = []
    for _ in range(2):
        c = c0.clone()
        assert mb.gemm(ta, tb, m, n, k, -1.25, a, lda, b, ldb, beta, c, ldc, mode=mode) == 0
        torch.cuda.synchronize()
        outs.append(c)
    err = (outs[0][:, :m].double().T - ref).abs().max() / ref.abs().max()
    assert err < tol_mode(mode, k)
    assert torch.equal(outs[0][:, m:], c0[:, m:]) and torch.equal(outs[0], outs[1])


@MODES
@pytest.mark.parametrize("uplo", ["L", "U"])
@pytest.mark.parametrize("beta", [0.0, 0.5])
@pytest.mark.parametrize("n,k", [(130, 4100), (700, 1000), (1025, 513)])
def test_split_syrk_few_tiles(mode, uplo, beta, n, k):
    torch = need_gpu()
    g = torch.Generator(device="cuda")
    g.manual_seed(n + k)
    a = torch.rand((k, n + 1), generator=g, device="cuda") * 2 - 1
    c0 = torch.rand((n, n + 3), generator=g, device="cuda") * 2 - 1
    c = c0.clone()
    assert mb.syrk(uplo, "N", n, k, 0.75, a, n + 1, beta, c, n + 3, mode=mode) == 0
    torch.cuda.synchronize()
    av = a[:, :n].double().T
    ref = 0.75 * av @ av.T + beta * c0[:, :n].double().T
    keep = torch.ones((n, n), device="cuda").tril().bool() if uplo == "L" else torch.ones((n, n), device="cuda").triu().bool()
    got = c[:, :n].double().T
    assert (got - ref)[keep].abs().max() / ref[keep].abs().max() < tol_mode(mode, k)
    assert torch.equal(c[:, :n].T[~keep], c0[:, :n].T[~keep]) and torch.equal(c[:, n:], c0[:, n:])
