"""Calls captured into a CUDA graph after a first call on the stream, with the cluster and dependent-launch attributes
their kernels take: a replay on new values gives the bits of the same calls made directly.  Each graph
holds a chain of calls, one reading what the one before wrote, on a stream that is not the default one."""
import pytest

import mojoblas_b200 as mb
from tests.gpu_util import need_gpu

pytestmark = pytest.mark.gpu


def run(torch, make, fill):
    """make() -> (call, outputs); fill() puts new values into the inputs."""
    mb.load()
    side = torch.cuda.Stream()
    try:
        with torch.cuda.stream(side):
            mb.set_stream(side)
            mb.set_sync(False)
            call, outputs = make()
            call()
            side.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=side):
                call()
            fill()
            graph.replay()
            side.synchronize()
            replayed = [o.clone() for o in outputs]
            for o in outputs:
                o.fill_(5.0)
            call()
            side.synchronize()
            for x, y in zip(replayed, outputs):
                assert torch.isfinite(y).all() and torch.equal(x, y)
    finally:
        mb.set_sync(True)
        mb.set_stream(None)


# shared tiles, whole tiles, stream-K, and the two Ozaki kernels (a triangle mask takes the single-CTA one)
GEMMS = [("f32", mb.PLAIN, 300, 200, 700), ("f32", mb.PLAIN, 2300, 2300, 64), ("f64", mb.PLAIN, 300, 200, 700),
         ("f64", mb.PLAIN, 2300, 2300, 64), ("f32", mb.BF16X6, 300, 400, 900), ("f32", mb.BF16X3, 300, 400, 900),
         ("f32", mb.BF16X6, 2560, 4096, 200), ("f64", mb.OZAKI, 400, 300, 500)]


@pytest.mark.parametrize("dt,mode,m,n,k", GEMMS)
def test_gemm_chain(dt, mode, m, n, k):
    torch = need_gpu()
    dtype = torch.float32 if dt == "f32" else torch.float64
    g = torch.Generator(device="cuda")
    g.manual_seed(9)
    a, b, e = (torch.empty(s, device="cuda", dtype=dtype) for s in ((k, m), (n, k), (m, n)))
    c, d = (torch.empty(s, device="cuda", dtype=dtype) for s in ((n, m), (m, m)))

    def fill():
        for t in (a, b, e):
            t.uniform_(-1, 1, generator=g)

    def make():
        fill()

        def call():  # C := A B, D := C E
            assert mb.gemm("N", "N", m, n, k, 1.5, a, m, b, k, 0.0, c, m, mode=mode) == 0
            assert mb.gemm("N", "N", m, m, n, 0.5, c, m, e, n, 0.0, d, m, mode=mode) == 0

        return call, [c, d]

    run(torch, make, fill)


@pytest.mark.parametrize("dt,mode", [("f32", mb.PLAIN), ("f32", mb.BF16X6), ("f64", mb.OZAKI)])
def test_syrk_then_trsm(dt, mode):
    torch = need_gpu()
    dtype = torch.float32 if dt == "f32" else torch.float64
    g = torch.Generator(device="cuda")
    g.manual_seed(10)
    n, k, r = 1100, 300, 260
    a, t, b = (torch.empty(s, device="cuda", dtype=dtype) for s in ((k, n), (n, n), (r, n)))
    c, x = torch.empty((n, n), device="cuda", dtype=dtype), torch.empty((r, n), device="cuda", dtype=dtype)

    def fill():
        a.uniform_(-1, 1, generator=g)
        b.uniform_(-1, 1, generator=g)
        t.uniform_(-1, 1, generator=g).div_(n).diagonal().add_(2.0)

    def make():
        fill()

        def call():  # C := A A^T (lower), X := T^-1 B
            c.zero_()
            assert mb.syrk("L", "N", n, k, 1.0, a, n, 0.0, c, n, mode=mode) == 0
            x.copy_(b)
            assert mb.trsm("L", "L", "N", "N", n, r, 1.0, t, n, x, n, mode=mode) == 0

        return call, [c, x]

    run(torch, make, fill)
