"""cg3mCgemm3mStridedBatchedEx on the GPU: one launch over the batch gives the
bytes of the calls one by one (the tensor-core launch runs unsplit along K, so
its yardstick is the single call with one K partition)."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def _run(cg3m, torch, dev, form, m, n, k, batch, ops, pad, engine, alpha, beta, seed):
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)

    def rnd(*shape):
        return torch.view_as_complex(torch.rand(*shape, 2, generator=gen, device=dev) * 2 - 1)

    ta, tb = ops
    ar, ac = (m, k) if ta in "NR" else (k, m)
    br, bc = (k, n) if tb in "NR" else (n, k)
    lda, ldb, ldc = ar + pad, br + pad, m + pad
    # one spare column between problems: strides that are not whole matrices
    A, B, C = rnd(batch, ac + 1, lda), rnd(batch, bc + 1, ldb), rnd(batch, n + 1, ldc)
    one = C.clone()
    h = cg3m.default_handle()
    opts = cg3m.cg3mOptions(cg3m.FORM[form], cg3m.ROUNDING["off"], 0, 0, cg3m.ENGINE[engine], 0)
    al, be = cg3m.cx(alpha), cg3m.cx(beta)
    st = cg3m.lib.cg3mCgemm3mStridedBatchedEx(
        h.h, cg3m.OP[ta], cg3m.OP[tb], m, n, k, ctypes.byref(al), cg3m.ptr(A), lda, A.stride(0), cg3m.ptr(B), ldb,
        B.stride(0), ctypes.byref(be), cg3m.ptr(C), ldc, C.stride(0), batch, ctypes.byref(opts))
    assert st == cg3m.SUCCESS
    for i in range(batch):
        h.cgemm3m(ta, tb, m, n, k, alpha, A[i], lda, B[i], ldb, beta, one[i], ldc, form=form, rounding="off",
                  engine=engine, k_partitions=1)
    torch.cuda.synchronize()
    return C, one


# one row tile over and under the pair tile, a partial column tile, K off the K-block
@pytest.mark.parametrize("form", ["tf32x3", "bf16x6", "bf16x9"])
@pytest.mark.parametrize("m,n,k,batch,ops,pad", [(129, 100, 65, 20, "NN", 0), (257, 129, 200, 12, "CT", 3),
                                                 (512, 384, 513, 9, "TR", 0), (300, 77, 31, 40, "RC", 1)])
def test_tensor_batch_is_the_unsplit_calls(cg3m, cuda, form, m, n, k, batch, ops, pad):
    import torch

    got, want = _run(cg3m, torch, cuda, form, m, n, k, batch, ops, pad, "packed", 0.7 - 0.2j, 0.25 + 0.5j, m + k)
    assert torch.equal(torch.view_as_real(got).view(torch.int32), torch.view_as_real(want).view(torch.int32))


@pytest.mark.parametrize("form", ["fp32", "tf32x3", "bf16x6"])
@pytest.mark.parametrize("m,n,k,batch,ops,pad", [(20, 33, 40, 30, "NC", 0), (128, 64, 96, 7, "TT", 5),
                                                 (260, 200, 150, 2, "NN", 0), (1, 1, 1, 3, "RR", 0)])
def test_batch_against_float64(cg3m, cuda, form, m, n, k, batch, ops, pad):
    """Whatever way the planner picks: FP32 error, and padding untouched.  The
    bound is that of K rounded three-product terms of magnitude <= 2 * 2 (each
    part of a sum below 2) accumulated in FP32: 3 k 4 k^0 2^-24 per part."""
    import torch

    got, _ = _run(cg3m, torch, cuda, form, m, n, k, batch, ops, pad, "auto", 1.0, 0.0, 3)
    gen = torch.Generator(device=cuda)
    gen.manual_seed(3)
    ta, tb = ops
    ar, ac = (m, k) if ta in "NR" else (k, m)
    br, bc = (k, n) if tb in "NR" else (n, k)

    def rnd(*shape):
        return torch.view_as_complex(torch.rand(*shape, 2, generator=gen, device=cuda) * 2 - 1)

    A, B, C = rnd(batch, ac + 1, ar + pad), rnd(batch, bc + 1, br + pad), rnd(batch, n + 1, m + pad)

    def op(x, o):
        x = x.mT if o in "TC" else x
        return x.conj() if o in "CR" else x

    X = op(A[:, :ac, :ar].mT.to(torch.complex128), ta)
    Y = op(B[:, :bc, :br].mT.to(torch.complex128), tb)
    want = (X @ Y).mT
    err = torch.view_as_real(got[:, :n, :m].to(torch.complex128) - want).abs().max().item()
    assert err <= 3 * k * 4 * k * 2.0 ** -24 + 1e-6
    assert torch.equal(torch.view_as_real(got[:, n:, :].resolve_conj()), torch.view_as_real(C[:, n:, :]))
    assert torch.equal(torch.view_as_real(got[:, :, m:].resolve_conj()), torch.view_as_real(C[:, :, m:]))
