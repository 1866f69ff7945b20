"""A batch whose outputs are later problems' operands runs in order."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


# C of problem i is A (or B) of problem i + 1; backwards; within padded columns
@pytest.mark.parametrize("form,n", [("fp32", 96), ("bf16x6", 160)])
@pytest.mark.parametrize("chained", ["A", "B"])
@pytest.mark.parametrize("backwards", [False, True])
def test_chained_batch_equals_the_calls_in_order(cg3m, cuda, form, n, chained, backwards):
    import torch

    batch, ld = 6, n + 5
    gen = torch.Generator(device=cuda)
    gen.manual_seed(n + backwards)

    def rnd(*shape):
        return torch.view_as_complex(torch.rand(*shape, 2, generator=gen, device=cuda) * 2 - 1)

    chain, other = rnd(batch + 1, n, ld), rnd(batch, n, ld)
    one = chain.clone()
    step = -1 if backwards else 1
    first = batch if backwards else 0

    def operands(buf, i):  # chained operand, other operand, output of problem i
        X, Y, C = buf[first + step * i], other[i], buf[first + step * (i + 1)]
        return (X, Y, C) if chained == "A" else (Y, X, C)

    h = cg3m.default_handle()
    opts = cg3m.cg3mOptions(cg3m.FORM[form], cg3m.ROUNDING["off"], 0, 0, 0, 0)
    al, be = cg3m.cx(0.1), cg3m.cx(0.5)
    strides = {"X": step * n * ld, "Y": n * ld}
    sa, sb = (strides["X"], strides["Y"]) if chained == "A" else (strides["Y"], strides["X"])
    A, B, C = operands(chain, 0)
    st = cg3m.lib.cg3mCgemm3mStridedBatchedEx(h.h, 0, 0, n, n, n, ctypes.byref(al), cg3m.ptr(A), ld, sa, cg3m.ptr(B),
                                              ld, sb, ctypes.byref(be), cg3m.ptr(C), ld, step * n * ld, batch,
                                              ctypes.byref(opts))
    assert st == cg3m.SUCCESS
    for i in range(batch):
        A, B, C = operands(one, i)
        h.cgemm3m("N", "N", n, n, n, 0.1, A, ld, B, ld, 0.5, C, ld, form=form, rounding="off")
    torch.cuda.synchronize()
    assert torch.equal(torch.view_as_real(chain).view(torch.int32), torch.view_as_real(one).view(torch.int32))
