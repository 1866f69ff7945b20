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
