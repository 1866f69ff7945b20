"""Outputs of an exact tile that the selection did not flag and that the exact
products cannot certify: the FP64 fallback recomputes them like flagged ones."""
import pytest

pytestmark = pytest.mark.gpu


# 2077: rows off the 16-row count tiles, flag words that cross columns
@pytest.mark.parametrize("form,n,ops", [("tf32x3", 2048, "NN"), ("bf16x6", 2077, "TN"), ("bf16x9", 2048, "NC")])
def test_unflagged_uncertified_outputs_are_recomputed(cg3m, cuda, form, n, ops):
    """op(A)'s first 128 rows are large (dense flags: the 256-row band's tiles
    are taken), the others small enough for no flag.  Elements 2^0 .. 2^-30
    apart round in the scaled integers, and real data make every imaginary part
    0, so no output of the small rows is certified.

    A recomputed output is one FP32 rounding of an FP64 sum: 2^-24 of it, plus
    the two FP64 sums' own rounding, n terms of 2^-53 of sum |a b| each."""
    import torch

    gen = torch.Generator(device=cuda)
    gen.manual_seed(n)

    def real(rows, cols):
        return torch.rand(rows, cols, generator=gen, device=cuda) * 10 - 5

    X, Y = real(n, n), real(n, n)  # op(A), op(B)
    X *= torch.exp2(-torch.randint(0, 31, (n, n), generator=gen, device=cuda).float())
    X[:128] = real(128, n) * 64
    X[128:] *= 2.0 ** -8

    def stored(M, op):  # column-major, so the tensor is the transpose of the stored matrix
        return (M.T if op == "N" else M).contiguous().to(torch.complex64)

    A, B = stored(X, ops[0]), stored(Y, ops[1])
    want = X.double() @ Y.double()
    slack = 2 * n * 2.0 ** -53 * (X.double().abs() @ Y.double().abs())
    band = slice(0, 256)

    def check(C):
        re, im = C.T.real.double(), C.T.imag
        assert bool((im[band] == 0).all())
        err = (re - want)[band].abs()
        assert bool((err <= 2.0 ** -24 * want[band].abs() + slack[band]).all())

    h = cg3m.Handle()
    nan = complex(float("nan"), float("nan"))
    C = torch.full((n, n), nan, dtype=torch.complex64, device=cuda)
    info = h.cgemm3m(ops[0], ops[1], n, n, n, 1.0, A, n, B, n, 0.0, C, n, form=form)
    assert info["rounding"] == 1
    stats = h.rounding_stats()
    bands = -(-n // 256)
    assert stats["exact_tiles"] == bands  # the first band of rows
    assert stats["flagged"] == 128 * n and stats["fallback_outputs"] >= 128 * n
    check(C)
    Ah, Bh = A.cpu().pin_memory(), B.cpu().pin_memory()
    Ch = torch.full((n, n), nan, dtype=torch.complex64).pin_memory()
    h.cgemm3m_host(ops[0], ops[1], n, n, n, 1.0, Ah, n, Bh, n, 0.0, Ch, n, form=form)
    assert h.rounding_stats() == stats
    check(Ch.to(cuda))
