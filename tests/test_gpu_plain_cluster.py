"""Plain float32 / float64 products whose reduction is shared by the CTAs of a cluster (few output
tiles): edges of tiles and of the slabs' division, every transpose pair, alignment and beta
form, and repeat calls with the same bits.  Tolerances: 1e-6 sqrt(k) and 4e-16 sqrt(k) of the
largest entry, those of the plain kernels' other tests, against float64 (float64 products:
torch's, within the same bound)."""
import numpy as np
import pytest

import mojoblas_b200 as mb
from tests.gpu_util import need_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", ["f32", "f64"])
@pytest.mark.parametrize("ta", ["N", "T"])
@pytest.mark.parametrize("tb", ["N", "T"])
@pytest.mark.parametrize("beta", [0.0, 1.0, 0.5])
@pytest.mark.parametrize("pad", [0, 3, 4])
@pytest.mark.parametrize("m,n,k", [(64, 64, 1000), (64, 64, 33), (65, 63, 17), (129, 257, 300), (512, 512, 512),
                                   (300, 521, 257), (96, 532, 95), (1000, 128, 1024)])
def test_plain_gemm_few_tiles(dt, ta, tb, beta, pad, m, n, k):
    torch = need_gpu()
    dtype, unit = (torch.float32, 1e-6) if dt == "f32" else (torch.float64, 4e-16)
    g = torch.Generator(device="cuda")
    g.manual_seed(m + n + k + pad)

    def uniform(*shape):
        return torch.rand(shape, generator=g, device="cuda", dtype=dtype) * 2 - 1

    lda, ldb, ldc = (m if ta == "N" else k) + pad, (k if tb == "N" else n) + pad, m + pad
    a, b, c0 = uniform(k if ta == "N" else m, lda), uniform(n if tb == "N" else k, ldb), uniform(n, ldc)
    av, bv = a[:, :lda - pad].double(), b[:, :ldb - pad].double()
    ref = -1.25 * (av.T if ta == "N" else av) @ (bv.T if tb == "N" else bv) + beta * c0[:, :m].double().T
    outs = []
    for _ in range(2):
        c = c0.clone()
        assert mb.gemm(ta, tb, m, n, k, -1.25, a, lda, b, ldb, beta, c, ldc) == 0
        torch.cuda.synchronize()
        outs.append(c)
    err = (outs[0][:, :m].double().T - ref).abs().max() / ref.abs().max()
    assert err < 2 * unit * np.sqrt(max(k, 16))
    assert torch.equal(outs[0][:, m:], c0[:, m:]) and torch.equal(outs[0], outs[1])
