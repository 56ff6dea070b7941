"""The step interpolates at 32-bit indices and spreads real gradients at the mirror pairs' integer ones: at
n = 256 the gradient with respect to the eigenvolumes and the one with respect to their log scales, which
follows the projections alone, agree to what that difference of positions allows."""
import pytest
import torch

pytestmark = pytest.mark.gpu

L = 128
# A 32-bit index is off by some 1.1e-6 of a radian (two products, their sum, the pixel's frequency and the
# wrap, of angles up to 4.4), 4.5e-5 cells, and 1.5e-5 cells for its own two roundings; a change of one cell
# along an axis turns the transform of a volume of L voxels by at most pi L / n of its norm.
TOL = 3**0.5 * 3.1416 * 0.5 * 6.0e-5


def _rotations(B, dev, g):
    return torch.linalg.qr(torch.randn((B, 3, 3), generator=g, device=dev, dtype=torch.float64))[0].float()


@pytest.mark.parametrize("disc", ["nufft", "bilinear"])
@pytest.mark.parametrize("objective", [0, 1])
def test_both_gradients_of_the_step(pkg, dev, disc, objective):
    r, B = 3, 6
    g = torch.Generator(device=dev).manual_seed(3)
    vec = torch.randn((r, L, L, L), generator=g, device=dev) / L
    logs = torch.randn((r,), generator=g, device=dev) * 0.3
    images = torch.randn((B, L * L), generator=g, device=dev, dtype=torch.complex64) * L
    step = pkg.FusedCovarStep(L, r, disc, 2, device=dev)
    step.set_rotations(_rotations(B, dev, g))
    _, gv, gl = step(vec, logs, images, torch.rand((B, L * L), generator=g, device=dev) + 0.3, 1.0e4, 0.0, None,
                     objective)
    v, gv, gl = vec.double().reshape(r, -1), gv.double().reshape(r, -1), gl.double()
    both = (v * gv).sum(1)
    assert ((both - gl).abs() <= TOL * v.norm(dim=1) * gv.norm(dim=1)).all()


@pytest.mark.parametrize("kernel,width", [(0, 6), (1, 0)])
def test_spreading_at_either_position(pkg, dev, kernel, width):
    B = 4
    g = torch.Generator(device=dev).manual_seed(4)
    plan = pkg.nufft_plan._Plan(L, 2, 1e-6, kernel, 2, width=width, device=dev)
    plan.setrot(_rotations(B, dev, g), L)
    vals = torch.randn((2, B * L * L), generator=g, device=dev, dtype=torch.complex64)
    flags = pkg._lib.APPLY_NYQUIST
    pairs = plan.backproject(vals, None, flags | pkg._lib.REAL_OUTPUT, 1.0).real.double()
    full = plan.backproject(vals, None, flags, 1.0).real.double()
    assert (pairs - full).norm() <= TOL * full.norm()
