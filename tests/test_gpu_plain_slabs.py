"""Plain float32 128-tiles at the edges of their k slabs, which are 16 or 32 deep by k and by the operands'
alignment: products and ssyrk against float64, 2e-6 sqrt(max(k, 16)) of the largest entry as for the
plain kernels' other tests."""
import numpy as np
import pytest

import mojoblas_b200 as mb
from tests.gpu_util import need_gpu

pytestmark = pytest.mark.gpu
KS = [1, 15, 16, 17, 31, 32, 33, 40, 48, 64, 65, 144, 160, 200]


def uniform(torch, g, *shape):
    return torch.rand(shape, generator=g, device="cuda") * 2 - 1


@pytest.mark.parametrize("pad_a,pad_b", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("ta,tb", [("N", "T"), ("N", "N"), ("T", "T")])
def test_gemm(ta, tb, pad_a, pad_b):
    torch = need_gpu()
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    m, n = 2180, 2300  # 18 x 18 tiles: more than two per SM
    for k in KS:
        lda, ldb = (m if ta == "N" else k) + pad_a, (k if tb == "N" else n) + pad_b
        a, b = uniform(torch, g, k if ta == "N" else m, lda), uniform(torch, g, n if tb == "N" else k, ldb)
        c = uniform(torch, g, n, m)
        av, bv = a[:, :lda - pad_a].double(), b[:, :ldb - pad_b].double()
        ref = 1.5 * (av.T if ta == "N" else av) @ (bv.T if tb == "N" else bv) - 0.5 * c.double().T
        assert mb.gemm(ta, tb, m, n, k, 1.5, a, lda, b, ldb, -0.5, c, m) == 0
        torch.cuda.synchronize()
        assert (c.double().T - ref).abs().max() / ref.abs().max() < 2e-6 * np.sqrt(max(k, 16)), k


@pytest.mark.parametrize("pad", [0, 1])
@pytest.mark.parametrize("trans", ["N", "T"])
def test_syrk(trans, pad):
    torch = need_gpu()
    g = torch.Generator(device="cuda")
    g.manual_seed(4)
    n = 700
    for k in KS:
        ld = (n if trans == "N" else k) + pad
        a = uniform(torch, g, k if trans == "N" else n, ld)
        c = torch.zeros((n, n), device="cuda")
        v = a[:, :ld - pad].double()
        v = v.T if trans == "N" else v
        ref = torch.tril(v @ v.T)
        assert mb.syrk("L", trans, n, k, 1.0, a, ld, 0.0, c, n) == 0
        torch.cuda.synchronize()
        assert (c.double().T - ref).abs().max() / ref.abs().max() < 2e-6 * np.sqrt(max(k, 16)), k
