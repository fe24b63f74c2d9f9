"""Grouped split sgemm plans take a reduction of 2^31 elements or more, as the single calls do.  The plan
is only built (its one tile would run for most of a minute; the slabs' arithmetic at such sizes is
checked by tests/test_schedule.py); with alpha == 0, where no operand is read, it runs."""
import ctypes as C

import pytest

from mojoblas_b200 import _lib as L
from tests.gpu_util import need_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [L.MODE_BF16X3, L.MODE_BF16X6], ids=["bf16x3", "bf16x6"])
@pytest.mark.parametrize("k", [2**31 - 1, 2**31, 2**31 + 64])
def test_plan_takes_long_reductions(mode, k):
    torch = need_gpu()
    lib = L.load()
    lib.mbg_set_stream(None)
    row = torch.empty(k, device="cuda")  # a row of op(A) and a column of op(B)
    c = torch.full((1,), 3.0, device="cuda")
    torch.cuda.synchronize()
    for alpha, run in ((1.0, False), (0.0, True)):
        probs = (L.SgemmProblem * 1)(L.SgemmProblem(b"N", b"N", 1, 1, k, alpha, 0.5, row.data_ptr(), 1, row.data_ptr(), k,
                                                    c.data_ptr(), 1))
        plan = C.c_void_p()
        assert lib.mbg_sgemm_grouped_plan(mode, 1, probs, C.byref(plan)) == 0, L.last_error()
        try:
            if run:
                assert lib.mbg_plan_execute(plan) == 0, L.last_error()
                torch.cuda.synchronize()
        finally:
            lib.mbg_plan_destroy(plan)
    assert c.item() == 1.5
