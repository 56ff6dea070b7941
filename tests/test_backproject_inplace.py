"""The real backprojection is a tensor of its own: it can be changed in place, with the gradients of that."""
import pytest
import torch


class _Doubling:
    """A plan whose backprojection and projection both double."""

    def backproject(self, values, ctf, flags, scale):
        return 2 * values.to(torch.complex64)

    project = backproject


@pytest.mark.parametrize("real", [False, True])
def test_in_place_change_of_the_result(pkg, real):
    from importlib import import_module

    fn = import_module("3dcovarestimation_gb300.nufft_plan")._BackprojectFn
    x = torch.arange(1.0, 5.0).reshape(1, 4).to(torch.complex64).requires_grad_()
    y = fn.apply(x, _Doubling(), None, 0, 1.0, real)
    assert y.is_complex() != real
    y *= 3
    (y if real else y.real).sum().backward()
    assert torch.equal(y.detach().real if not real else y.detach(), 6 * x.detach().real)
    assert torch.equal(x.grad.real, torch.full((1, 4), 6.0))
