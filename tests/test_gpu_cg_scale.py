"""The CG's inner products have the range of FP64: a right side scaled by a power of two far from one
gives the iterates scaled by it (every other operation is exact under such a scale)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precond", [None, "diagonal", "circulant"])
@pytest.mark.parametrize("L", [24, 32, 64])  # cuFFT, fused axis 0, line kernels
@pytest.mark.parametrize("exponent", [-70, 66])
def test_scaled_right_side(pkg, dev, L, precond, exponent):
    n = 2 * L
    g = torch.Generator(device=dev).manual_seed(L)
    ax = torch.arange(n, device=dev) - n // 2
    k2 = (ax[:, None, None] ** 2 + ax[None, :, None] ** 2 + ax[None, None, :] ** 2).float()
    reg = (1.0 + 40.0 / (1.0 + k2) + k2 / n**2 + 0.1 * torch.rand((n, n, n), generator=g, device=dev)).contiguous()
    b = torch.randn((L, L, L), generator=g, device=dev).to(torch.complex64)
    x0 = torch.zeros_like(b)
    s = 2.0**exponent
    want, a = pkg.cg_solve(reg, b, x0, L, rtol=1e-4, maxiter=40, precond=precond, history=True)
    got, c = pkg.cg_solve(reg, b * s, x0, L, rtol=1e-4, maxiter=40, precond=precond, history=True)
    assert a.converged and c.converged and a.iters == c.iters
    # the sums' order (atomics) is all that differs: scalars to some 1e-15, the float steps made of them now
    # and then by one rounding, 6e-8, in each of at most 40 iterations
    assert (got / s - want).norm() < 40 * 6e-8 * want.norm()
