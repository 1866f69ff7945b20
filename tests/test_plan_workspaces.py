"""No call takes more than a default workspace (32 MiB) that did with less, and
no split more than an eighth over a larger one (host only; the allocation-free
entry point on the GPU).  The golden sizes are those of the K-split rule's own
plans (csrc/chains.cpp)."""
import ctypes
import json
import os

import pytest

with open(os.path.join(os.path.dirname(__file__), "golden", "plan_workspaces.json")) as f:
    GOLDEN = json.load(f)
DEFAULT = 32 << 20


def test_products(cg3m):
    for m, n, k, rule in GOLDEN["product"]:
        got = cg3m.plan("N", "N", m, n, k, alpha=0.5)["workspace_bytes"]
        assert got <= (DEFAULT - 256 if rule <= DEFAULT - 256 else rule * 9 / 8), (m, n, k)


def test_strided_batches(cg3m):
    for m, n, k, mode, batch, rule in GOLDEN["onchip"]:
        # the tile counters of another tile shape besides (4 bytes per 32 x 32 tile)
        counters = 4 * batch * -(-m // 32) * -(-n // 32) + 512
        got = cg3m.plan_onchip(m, n, k, mode, batch)["workspace_bytes"]
        assert got <= max(DEFAULT, rule + counters), (m, n, k, batch)


# packed plans beyond the array: once one-launch plans, or faster as such
@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(1864, 40, 1765), (28, 369, 8510), (531, 25, 6770), (1592, 51, 1814), (46, 786, 9358)])
def test_allocation_free_call_takes_the_one_launch_engine(cg3m, cuda, m, n, k):
    import torch

    gen = torch.Generator(device=cuda)
    gen.manual_seed(k)
    A, B = (torch.view_as_complex(torch.rand(*s, 2, generator=gen, device=cuda) * 2 - 1) for s in ((k, m), (n, k)))
    C = torch.zeros(n, m, dtype=torch.complex64, device=cuda)
    al, be = cg3m.cx(1.0), cg3m.cx(0.0)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    st = cg3m.lib.cg3mCgemm3mNoAlloc(stream, 0, 0, m, n, k, ctypes.byref(al), cg3m.ptr(A), m, cg3m.ptr(B), k,
                                     ctypes.byref(be), cg3m.ptr(C), m)
    assert st == cg3m.SUCCESS
    want = (A.T.to(torch.complex128) @ B.T.to(torch.complex128)).T
    # FP32 chains of at most k / 8 + 16 terms, 3 products, errors of both signs:
    # 2.6e-8 sqrt(terms) of the norm on uniform data, 1.5 times that allowed
    err = float((C.to(torch.complex128) - want).norm() / want.norm())
    assert err <= 1.5 * 2.6e-8 * (k / 8 + 16) ** 0.5
