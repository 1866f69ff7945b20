"""Host-buffer panels that would pass the rounding pass's gate by themselves."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["fp32", "bf16x6"])
def test_square_panels_of_a_wide_product_run_no_pass(cg3m, cuda, form):
    """Two 2048^3 panels: the whole product, 4096 columns, is not square, so its
    device call runs no rounding pass and neither does a panel."""
    import torch

    m = k = 2048
    n = 2 * m
    gen = torch.Generator(device=cuda)
    gen.manual_seed(5)
    A, B = (torch.view_as_complex(torch.rand(c, r, 2, generator=gen, device=cuda) * 200 - 100) for c, r in ((k, m), (n, k)))
    C = torch.zeros(n, m, dtype=torch.complex64, device=cuda)
    h = cg3m.Handle()
    assert h.cgemm3m("N", "N", m, n, k, 1.0, A, m, B, k, 0.0, C, m, form=form)["rounding"] == 0
    Ch = torch.zeros(n, m, dtype=torch.complex64).pin_memory()
    info = h.cgemm3m_host("N", "N", m, n, k, 1.0, A.cpu().pin_memory(), m, B.cpu().pin_memory(), k, 0.0, Ch, m,
                          form=form, panels=2)
    assert info["rounding"] == 0
    assert torch.equal(torch.view_as_real(Ch).view(torch.int32), torch.view_as_real(C.cpu()).view(torch.int32))
