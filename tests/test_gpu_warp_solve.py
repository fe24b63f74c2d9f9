"""Grouped strsm at the edges of its 32-row blocks and 32-column strips, against a float64 solve
(the inversion of diagonal blocks by the same routine: tests/test_gpu_trsm_inverse.py).

Tolerance: an entry of X is rounded at its own size once for alpha B, once for the sum of
the earlier blocks, at most 31 times within its diagonal block and twice for the
reciprocal and its multiply: a random walk of 35 half-ulp roundings, whose four-sigma
point is 7 eps of the largest entry."""
import ctypes as C

import numpy as np
import pytest

from mojoblas_b200 import _lib as L

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float32).eps


def triangle(torch, g, n, ld, uplo, diag):
    """n x n with ld >= n, the other triangle (and for a unit diagonal the diagonal) 1e30: never used."""
    a = torch.full((n, ld), 1e30, device="cuda")
    t = torch.randn((n, n), generator=g, device="cuda", dtype=torch.float64) / n ** 0.5
    if diag == "U":
        t /= n
    m = t.T.clone()  # M(i, j) = a[j, i]
    m.diagonal().copy_(n + torch.rand(n, generator=g, device="cuda", dtype=torch.float64))
    m = (torch.tril(m) if uplo == "L" else torch.triu(m)).float().double()
    keep = torch.ones((n, n), device="cuda").tril().bool() if uplo == "L" else torch.ones((n, n), device="cuda").triu().bool()
    if diag == "U":
        keep = keep & ~torch.eye(n, device="cuda").bool()
        m.diagonal().fill_(1.0)
    a[:, :n] = torch.where(keep, m, torch.full_like(m, 1e30)).T.float()
    return a, m


@pytest.mark.parametrize("pad,off", [(0, 0), (3, 1), (4, 0)], ids=["tight", "odd", "vec16"])
@pytest.mark.parametrize("diag", ["N", "U"])
@pytest.mark.parametrize("ta", ["N", "T"])
@pytest.mark.parametrize("uplo", ["L", "U"])
def test_grouped_strsm_edges(uplo, ta, diag, pad, off):
    torch = pytest.importorskip("torch")
    lib = L.load()
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    sizes = [(n, r) for n in (1, 8, 31, 32, 33, 64, 65, 97, 128, 160, 224, 255, 256) for r in (1, 31, 32, 33, 64)]
    probs, held = (L.StrsmProblem * len(sizes))(), []
    for i, (n, r) in enumerate(sizes):
        ld = (n + 3) // 4 * 4 + pad if pad == 4 else n + pad
        a, m = triangle(torch, g, n, ld, uplo, diag)
        buf = torch.empty(n * ld + off, device="cuda")
        buf[off:] = a.reshape(-1)
        b = torch.randn(r * ld + off, generator=g, device="cuda")
        held.append((buf, b, b.clone(), m, n, r, ld))
        probs[i] = L.StrsmProblem(b"L", uplo.encode(), ta.encode(), diag.encode(), n, r, 1.5, buf.data_ptr() + 4 * off,
                                  ld, b.data_ptr() + 4 * off, ld)
    plan = C.c_void_p()
    torch.cuda.synchronize()
    assert lib.mbg_strsm_grouped_plan(L.MODE_PLAIN, len(sizes), probs, C.byref(plan)) == 0, L.last_error()
    try:
        assert lib.mbg_plan_execute(plan) == 0, L.last_error()
        torch.cuda.synchronize()
        for buf, b, b0, m, n, r, ld in held:
            got, was = b[off:].view(r, ld), b0[off:].view(r, ld)
            op = m if ta == "N" else m.T
            x = torch.linalg.solve_triangular(op, 1.5 * was[:, :n].double().T, upper=(uplo == "U") == (ta == "N"))
            err = (got[:, :n].double().T - x).abs().max() / x.abs().max()
            assert err < 8 * EPS, (n, r, float(err))
            assert torch.equal(got[:, n:], was[:, n:]), (n, r)  # what lies between the columns stays
    finally:
        lib.mbg_plan_destroy(plan)


def test_grouped_strsm_zero_pivots():
    """A zero of X takes part in nothing, whatever its column of op(A) holds (infinities and a zero
    diagonal here), within its 32-row block and in the later ones."""
    torch = pytest.importorskip("torch")
    lib = L.load()
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    n, r = 200, 40
    a, m = triangle(torch, g, n, n, "L", "N")
    b = torch.randn((r, n), generator=g, device="cuda")
    hole = [0, 5, 40, 100, 131]
    a[:, :] = torch.where(torch.ones((n, n), device="cuda").triu().bool(), a, torch.zeros_like(a))  # a[l, i] = A(i, l)
    for h in hole:  # row h of A is its diagonal alone, so x_h = b_h / a_hh, and b_h = 0
        a[:h, h] = 0.0
        m[h, :h] = 0.0
        b[:, h] = 0.0
        a[h, h:] = float("inf")
        a[h, h] = 0.0
        m[h:, h] = 0.0
        m[h, h] = 1.0
    x = torch.linalg.solve_triangular(m, b.double().T, upper=False)
    probs = (L.StrsmProblem * 1)(L.StrsmProblem(b"L", b"L", b"N", b"N", n, r, 1.0, a.data_ptr(), n, b.data_ptr(), n))
    torch.cuda.synchronize()
    assert lib.mbg_strsm_grouped(L.MODE_PLAIN, 1, probs) == 0, L.last_error()
    torch.cuda.synchronize()
    assert (b.double().T - x).abs().max() / x.abs().max() < 8 * EPS
    assert (b[:, hole] == 0).all()
