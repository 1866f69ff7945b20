"""The host-buffer entry point with the rounding pass in a tensor-core form
runs panel by panel: the bytes and the pass's counters of the device call."""
import pytest

pytestmark = pytest.mark.gpu


# 2048: panels of two tiles; 2077: flag words that cross columns, a ragged last
# panel; 2304: an odd number of tile columns
@pytest.mark.parametrize("form,n,ops,panels", [("bf16x6", 2077, "TC", 0), ("tf32x3", 2304, "NN", 0),
                                               ("bf16x9", 2048, "CT", 3), ("bf16x6", 2304, "NT", 1)])
def test_panels_equal_the_device_call(cg3m, cuda, form, n, ops, panels):
    import torch

    gen = torch.Generator(device=cuda)
    gen.manual_seed(n)

    def rnd(scaled, axis):
        x = torch.view_as_complex(torch.rand(n, n, 2, generator=gen, device=cuda) * 10 - 5)
        # a band of large rows of op(A) and columns of op(B): tiles with dense
        # flags beside tiles with a few and tiles with none
        x.narrow(axis, *scaled).mul_(8)
        return x

    # stored column-major, so the tensor's rows are the matrix's columns
    A = rnd((0, 700), 1 if ops[0] == "N" else 0)
    B = rnd((600, 900), 0 if ops[1] == "N" else 1)
    h = cg3m.Handle()
    C = torch.zeros(n, n, dtype=torch.complex64, device=cuda)
    info = h.cgemm3m(ops[0], ops[1], n, n, n, 1.0, A, n, B, n, 0.0, C, n, form=form)
    assert info["rounding"] == 1
    want = h.rounding_stats()
    assert want["exact_tiles"] > 0 and want["sparse_outputs"] > 0 and want["exact_positions"] < n * n
    Ah, Bh = A.cpu().pin_memory(), B.cpu().pin_memory()
    Ch = torch.zeros(n, n, dtype=torch.complex64).pin_memory()
    for _ in range(2):  # the second call reuses the device copies and the workspace
        Ch.zero_()
        got = h.cgemm3m_host(ops[0], ops[1], n, n, n, 1.0, Ah, n, Bh, n, 0.0, Ch, n, form=form, panels=panels)
        assert got["rounding"] == 1 and got["k_partitions"] == 1
        assert h.rounding_stats() == want
        assert torch.equal(torch.view_as_real(Ch).view(torch.int32), torch.view_as_real(C.cpu()).view(torch.int32))
