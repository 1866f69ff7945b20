"""One launch over a batch is as accurate as the calls one by one."""
import pytest

pytestmark = pytest.mark.gpu


# shapes whose single calls run finely split FP32 chains (16 terms and up), a
# long K, an unsplit FP32 call, and two that run the tensor-core form
@pytest.mark.parametrize("form,m,n,k,batch", [
    ("bf16x6", 162, 822, 188, 8), ("bf16x6", 822, 188, 162, 8), ("tf32x3", 378, 217, 281, 4), ("fp32", 140, 303, 580, 16),
    ("fp32", 328, 203, 140, 8), ("fp32", 133, 195, 3000, 6), ("fp32", 971, 968, 407, 4), ("bf16x6", 788, 660, 385, 8),
    ("tf32x3", 1024, 512, 1024, 4),
])
def test_batch_error_is_the_single_calls(cg3m, cuda, form, m, n, k, batch):
    """Relative to the Frobenius norm, over at least 10^5 outputs, the error of a
    chain length repeats within a few per cent on new data, and a tensor-core
    form's changes by at most 5 % with the K split: 10 % are allowed."""
    import torch

    gen = torch.Generator(device=cuda)
    gen.manual_seed(m + n + k)

    def rnd(*shape):
        return torch.view_as_complex(torch.rand(*shape, 2, generator=gen, device=cuda) * 2 - 1)

    A, B = rnd(batch, m, k), rnd(batch, k, n)
    want = A.to(torch.complex128) @ B.to(torch.complex128)

    def error(C):
        return float((C.to(torch.complex128) - want).norm() / want.norm())

    one = torch.stack([cg3m.cgemm3m(A[i], B[i], form=form, rounding="off") for i in range(batch)])
    assert error(cg3m.cgemm3m_batched(A, B, form=form)) <= 1.1 * error(one)
