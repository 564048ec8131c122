"""The views that YeeSolver.fields hands out are ordinary single views of the state."""
import pytest
import torch


def test_fields_take_writes_that_autograd_records():
    from fdtd_accelerate_gb300.solver import YeeSolver
    s = YeeSolver((6, 7, 9), device="cpu")
    w = torch.full((6, 7, 9), 2.0, requires_grad=True)
    s.set_fields(ex=w)
    s.fields["hy"].copy_(3.0 * w)
    assert torch.equal(s.fields["ex"].detach(), w.detach()) and torch.equal(s.fields["hy"].detach(), 3.0 * w.detach())
    assert s.fields["ez"].stride() == (7 * 12, 12, 1)


@pytest.mark.parametrize("nz", [8, 9])
def test_symplectic_fields_and_coefficients(nz):
    from fdtd_accelerate_gb300.symplectic import SymplecticSolver
    w = torch.full((6, 7, nz), 0.5, requires_grad=True)
    s = SymplecticSolver((6, 7, nz), ce=[w] * 3, ch=[w] * 3, device="cpu")
    assert s.fields["ex"].is_contiguous() and s.ce[0].data_ptr() == w.data_ptr() and s.ch[2].data_ptr() == w.data_ptr()


@pytest.mark.parametrize("nz", [8, 9])
def test_symplectic_coefficients_of_too_few_elements(nz):
    from fdtd_accelerate_gb300.symplectic import SymplecticSolver
    full = torch.zeros(6 * 7 * nz)
    for bad in (torch.zeros(nz), torch.zeros(6, 7, nz - 1), 0.5):
        for kw in ({"ce": [full, full, bad]}, {"ch": [bad, full, full]}):
            with pytest.raises(ValueError, match="fewer elements"):
                SymplecticSolver((6, 7, nz), device="cpu", **kw)
    SymplecticSolver((6, 7, nz), ce=[full] * 3, ch=[full.view(6, 7, nz)] * 3, device="cpu")
