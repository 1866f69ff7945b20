"""cg3mCgemm3mStridedBatchedEx bit for bit: the FP32 launch against single
calls, and the tensor-core launch in chunks of problems."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def _rnd(torch, device, *shape, seed):
    gen = torch.Generator(device=device)
    gen.manual_seed(seed)
    return torch.view_as_complex(torch.rand(*shape, 2, generator=gen, device=device) * 2 - 1)


def _batch(cg3m, h, A, B, C, m, n, k, form, engine="auto"):
    """Column-major A (batch, k, m), B (batch, n, k), C (batch, n, m); the status."""
    al, be = cg3m.cx(0.75 + 0.25j), cg3m.cx(0.0)
    opts = cg3m.cg3mOptions(cg3m.FORM[form], cg3m.ROUNDING["off"], 0, 0, cg3m.ENGINE[engine], 0)
    return cg3m.lib.cg3mCgemm3mStridedBatchedEx(
        h.h, 0, 0, m, n, k, ctypes.byref(al), cg3m.ptr(A), m, m * k, cg3m.ptr(B), k, k * n, ctypes.byref(be),
        cg3m.ptr(C), m, m * n, A.shape[0], ctypes.byref(opts))


def _singles(cg3m, torch, A, B, m, n, k, **kw):
    C = torch.empty(A.shape[0], n, m, dtype=torch.complex64, device=A.device)
    h = cg3m.default_handle()
    for i in range(A.shape[0]):
        h.cgemm3m("N", "N", m, n, k, 0.75 + 0.25j, A[i], m, B[i], k, 0.0, C[i], m, rounding="off", **kw)
    return C


def _same(torch, x, y):
    return torch.equal(torch.view_as_real(x).view(torch.int32), torch.view_as_real(y).view(torch.int32))


# small and many, a split chain, tiles with remainders, one row, many partitions
@pytest.mark.parametrize("m,n,k,batch", [(20, 33, 40, 30), (200, 260, 150, 12), (162, 188, 822, 8), (1, 70, 300, 16),
                                         (257, 31, 513, 9)])
def test_fp32_launch_is_the_single_calls_of_one_split(cg3m, cuda, m, n, k, batch):
    """Every output is a fixed function of the inputs and the K split, so the
    launch equals the single calls of some split, all problems alike."""
    import torch

    A, B = _rnd(torch, cuda, batch, k, m, seed=m), _rnd(torch, cuda, batch, n, k, seed=n)
    C = torch.full((batch, n, m), float("nan"), dtype=torch.complex64, device=cuda)
    assert _batch(cg3m, cg3m.default_handle(), A, B, C, m, n, k, "fp32") == cg3m.SUCCESS
    splits = range(1, min(32, -(-k // 16)) + 1)
    assert any(_same(torch, C, _singles(cg3m, torch, A, B, m, n, k, engine="packed", k_partitions=q)) for q in splits)


def test_more_problems_than_one_launch_holds(cg3m, cuda):
    """33 problems of 37.7 MB of operand planes: launches of 17 and 16."""
    import torch

    m = n = k = 1024
    A, B = _rnd(torch, cuda, 33, k, m, seed=1), _rnd(torch, cuda, 33, n, k, seed=2)
    C = torch.full((33, n, m), float("nan"), dtype=torch.complex64, device=cuda)
    h = cg3m.Handle(stream=torch.cuda.current_stream().cuda_stream)
    assert _batch(cg3m, h, A, B, C, m, n, k, "bf16x6", "packed") == cg3m.SUCCESS
    assert _same(torch, C, _singles(cg3m, torch, A, B, m, n, k, form="bf16x6", engine="packed", k_partitions=1))


# 9 problems of 8.4 MB of planes: allocations for 9, 5, 3, 2 and 1 of them fail
@pytest.mark.parametrize("failures,status", [(1, 0), (3, 0), (4, 0), (5, 4)])
def test_chunks_shrink_when_allocations_fail(cg3m, cuda, failures, status):
    import torch

    m, n, k = 512, 384, 513
    A, B = _rnd(torch, cuda, 9, k, m, seed=3), _rnd(torch, cuda, 9, n, k, seed=4)
    h = cg3m.Handle(stream=torch.cuda.current_stream().cuda_stream)
    h.cgemm3m("N", "N", 8, 8, 8, 1.0, A, 8, B, 8, 0.0, torch.empty(64, dtype=torch.complex64, device=cuda), 8)
    C = torch.full((9, n, m), float("nan"), dtype=torch.complex64, device=cuda)
    cg3m.lib.cg3mDiagFailAllocations(failures)
    try:
        st = _batch(cg3m, h, A, B, C, m, n, k, "bf16x6", "packed")
    finally:
        cg3m.lib.cg3mDiagFailAllocations(0)
    assert st == status
    if status != 0:  # and the handle recovers
        assert _batch(cg3m, h, A, B, C, m, n, k, "bf16x6", "packed") == cg3m.SUCCESS
    assert _same(torch, C, _singles(cg3m, torch, A, B, m, n, k, form="bf16x6", engine="packed", k_partitions=1))
