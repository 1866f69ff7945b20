"""Options out of range are refused the same way by every path (host only)."""
import ctypes

import pytest


@pytest.mark.parametrize("form", [-1, 4, 99, 1 << 20])
def test_planner_refuses_unknown_forms(cg3m, form):
    info = cg3m.cg3mCallInfo()
    opts = cg3m.cg3mOptions(form, 0, 0, 0, 0, 0)
    st = cg3m.lib.cg3mPlan(0, 0, 300, 200, 100, ctypes.byref(cg3m.cx(1)), 300, 100, ctypes.byref(cg3m.cx(0)), 300,
                           ctypes.byref(opts), 148, ctypes.byref(info))
    assert st == cg3m.INVALID_VALUE


@pytest.mark.parametrize("batch", [1, 3])
@pytest.mark.parametrize("rounding,parts", [(2, 0), (-1, 0), (0, -1), (7, 2)])
def test_batched_call_refuses_what_the_single_call_does(cg3m, rounding, parts, batch):
    """Refused before any device is touched, as cg3mCgemm3mEx refuses it."""
    h = ctypes.c_void_p()
    assert cg3m.lib.cg3mCreate(ctypes.byref(h)) == cg3m.SUCCESS
    opts = cg3m.cg3mOptions(0, rounding, parts, 0, 0, 0)
    al, be = cg3m.cx(1), cg3m.cx(0)
    x = ctypes.c_void_p(1 << 20)  # never read
    st = cg3m.lib.cg3mCgemm3mStridedBatchedEx(h, 0, 0, 8, 8, 8, ctypes.byref(al), x, 8, 64, x, 8, 64, ctypes.byref(be),
                                              x, 8, 64, batch, ctypes.byref(opts))
    assert st == cg3m.INVALID_VALUE
    cg3m.lib.cg3mDestroy(h)
