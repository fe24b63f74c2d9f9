"""A zero of X takes part in nothing, whatever its column of op(A) holds (infinities and a zero diagonal here): grouped
strsm in every orientation, within a 32-row block and across blocks (tests/test_gpu_warp_solve.py has the
lower, untransposed one)."""
import ctypes as C

import numpy as np
import pytest

from mojoblas_b200 import _lib as L
from tests.gpu_util import need_gpu

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float32).eps


@pytest.mark.parametrize("uplo,ta", [("L", "N"), ("L", "T"), ("U", "N"), ("U", "T")])
@pytest.mark.parametrize("n", [30, 64, 200, 256])
def test_zeros_of_x(uplo, ta, n):
    torch = need_gpu()
    lib = L.load()
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    r = 40
    lower = (uplo == "L") == (ta == "N")  # op(A)
    t = torch.randn((n, n), generator=g, device="cuda", dtype=torch.float64) / n ** 0.5
    t.diagonal().copy_(n + torch.rand(n, generator=g, device="cuda", dtype=torch.float64))
    t = (torch.tril(t) if lower else torch.triu(t)).float().double()  # op(A)
    b = torch.randn((r, n), generator=g, device="cuda")
    op = t.clone()
    for h in [h for h in (0, 5, 29, 31, 40, 63, 100, 131, 255) if h < n]:
        b[:, h] = 0.0
        t[h, :] = 0.0  # x_h = b_h / t_hh = 0
        t[:, h] = 0.0
        t[h, h] = 1.0
        op[h, :] = 0.0
        op[:, h] = torch.where(op[:, h] != 0, torch.full_like(op[:, h], float("inf")), op[:, h])
        op[h, h] = 0.0
    x = torch.linalg.solve_triangular(t, b.double().T, upper=not lower)
    a = (op.T if ta == "N" else op).float().contiguous()  # column-major A
    probs = (L.StrsmProblem * 1)(L.StrsmProblem(b"L", uplo.encode(), ta.encode(), b"N", n, r, 1.0, a.data_ptr(), n,
                                                b.data_ptr(), n))
    torch.cuda.synchronize()
    assert lib.mbg_strsm_grouped(L.MODE_PLAIN, 1, probs) == 0, L.last_error()
    torch.cuda.synchronize()
    assert (b.double().T - x).abs().max() / x.abs().max() < 8 * EPS  # tests/test_gpu_warp_solve.py has the bound
