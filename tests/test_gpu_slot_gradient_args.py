"""KuboPlan.slot_gradient refuses a matrix of another shape or device (its kernels take plain pointers) and
takes other strides and types."""
import pytest

pytestmark = pytest.mark.gpu


def test_slot_gradient_checks_its_matrix(cuda_lib):
    import torch

    from minijclsquant_gb300 import adjoint

    plan = adjoint.KuboPlan(5, 4, 18, R=1, n_energies=7)
    C = torch.randn((18, 18), dtype=torch.float64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    for bad in (C[:17], C[:, :17], C.reshape(-1), C[None], torch.zeros((19, 19), device="cuda"), C.cpu()):
        with pytest.raises((ValueError, RuntimeError)):
            plan.slot_gradient(bad)
    want = plan.slot_gradient(C)
    wide = torch.zeros((18, 40), dtype=torch.float64, device="cuda")
    wide[:, 3:21] = C
    assert torch.equal(plan.slot_gradient(wide[:, 3:21]), want)
    assert torch.equal(plan.slot_gradient(C.t().contiguous().t()), want)
    half = C.to(torch.float32)
    assert torch.equal(plan.slot_gradient(half), plan.slot_gradient(half.double()))
