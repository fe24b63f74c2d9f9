"""Calls that follow one another on a stream take no longer than the same call by itself: blocks of a call that
start beside those of the one before must not crowd the SMs those leave free.  (Such calls took 1.8 times
as long; the bound is 1.3, and a call by itself is timed with its launch.)"""
import pytest

import mojoblas_b200 as mb
from tests.gpu_util import need_gpu

pytestmark = pytest.mark.gpu


def shortest(torch, call, calls):
    call()
    torch.cuda.synchronize()
    best = float("inf")
    for _ in range(10):
        start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        start.record()
        for _ in range(calls):
            call()
        end.record()
        torch.cuda.synchronize()
        best = min(best, start.elapsed_time(end) / calls)
    return best


@pytest.mark.parametrize("what", ["sgemm", "ssyrk"])
def test_calls_in_a_row(what):
    torch = need_gpu()
    mb.load()
    mb.set_stream(torch.cuda.current_stream())
    mb.set_sync(False)
    try:
        if what == "sgemm":  # 64 tiles of 128 x 128
            a, b, c = (torch.rand((1000, 1000), device="cuda") for _ in range(3))
            call = lambda: mb.gemm("N", "T", 1000, 1000, 1000, 1.0, a, 1000, b, 1000, 0.0, c, 1000)
        else:  # 78 of them
            a, c = torch.rand((500, 1500), device="cuda"), torch.rand((1500, 1500), device="cuda")
            call = lambda: mb.syrk("L", "N", 1500, 500, 1.0, a, 1500, 0.0, c, 1500)
        assert shortest(torch, call, 50) < 1.3 * shortest(torch, call, 1)
    finally:
        mb.set_sync(True)
        mb.set_stream(None)
