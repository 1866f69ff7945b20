"""torch operands: lazy conjugate and negative views, and types that are refused."""
import itertools

import pytest


@pytest.fixture
def gpu(cg3m, cuda):
    return cuda


def _rnd(torch, device, *shape, seed=0):
    gen = torch.Generator(device=device)
    gen.manual_seed(seed)
    return torch.view_as_complex(torch.rand(*shape, 2, generator=gen, device=device) * 2 - 1)


def _lazy(torch, x):
    """The same values as views that torch resolves on reading: conjugate,
    conjugate of a transpose, negative."""
    return {"conj": x.conj().resolve_conj().conj(), "conj_t": x.mT.contiguous().conj().resolve_conj().mT.conj(),
            "neg": torch._neg_view(x)}


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["conj", "conj_t", "neg"])
@pytest.mark.parametrize("batch", [0, 3])
def test_lazy_views_are_resolved(cg3m, gpu, kind, batch):
    import torch
    from cg3m.autograd import cgemm3m_autograd

    lead = (batch,) if batch else ()
    A, B = (_lazy(torch, _rnd(torch, gpu, *lead, *s, seed=i))[kind] for i, s in enumerate([(40, 33), (33, 50)]))
    assert A.is_conj() or A.is_neg()
    want = A.to(torch.complex128) @ B.to(torch.complex128)
    # 33 terms of three FP32 products of magnitude <= 2 (a sum's parts), each
    # rounded once and added with one rounding: 3 * 33 * 2 * 33 * 2^-24 at most
    bound = 3 * 33 * 2 * 33 * 2.0 ** -24
    calls = [cgemm3m_autograd(A, B)]
    calls.append(cg3m.cgemm3m_batched(A, B) if batch else cg3m.cgemm3m(A, B))
    for got in calls:
        assert float((got.to(torch.complex128) - want).abs().max()) <= bound


@pytest.mark.gpu
def test_gradient_of_a_conjugated_output(cg3m, gpu):
    """The gradient that reaches the backward is a lazy conjugate."""
    import torch
    from cg3m.autograd import cgemm3m_autograd

    for lead in ((), (3,)):
        A, B = _rnd(torch, gpu, *lead, 40, 33, seed=1).requires_grad_(), _rnd(torch, gpu, *lead, 33, 50, seed=2)
        W = _rnd(torch, gpu, *lead, 40, 50, seed=3)
        (got,) = torch.autograd.grad((cgemm3m_autograd(A, B).conj() * W).sum().real, A)
        wide = A.detach().to(torch.complex128).requires_grad_()
        (want,) = torch.autograd.grad(((wide @ B.to(torch.complex128)).conj() * W).sum().real, wide)
        assert float((got.to(torch.complex128) - want).abs().max()) <= 3 * 50 * 2 * 50 * 2.0 ** -24


@pytest.mark.gpu
def test_beta_reads_a_lazy_output(cg3m, gpu):
    import torch

    A, B, C = (_rnd(torch, gpu, *s, seed=i) for i, s in enumerate([(20, 16), (16, 24), (20, 24)]))
    got = cg3m.cgemm3m(A, B, beta=1.0, C=C.clone().conj())
    want = A.to(torch.complex128) @ B.to(torch.complex128) + C.conj().to(torch.complex128)
    assert float((got.to(torch.complex128) - want).abs().max()) <= 3 * 16 * 2 * 17 * 2.0 ** -24


@pytest.mark.gpu
@pytest.mark.parametrize("types", list(itertools.product(["complex64", "complex128", "float32"], repeat=2))[1:])
def test_other_types_are_refused(cg3m, gpu, types):
    """The library reads 8 bytes an element, whatever the tensor holds."""
    import torch

    A, B = (torch.ones(2, 8, 8, dtype=getattr(torch, t), device=gpu) for t in types)
    for call in (lambda: cg3m.cgemm3m_batched(A, B), lambda: cg3m.cgemm3m(A[0], B[0])):
        with pytest.raises(TypeError):
            call()
