"""Linear spreading at the channel counts where its layouts change (passes of twelve, then 7-8, 3-6, two,
one), against 64-bit sums over the interpolation's weights; a real volume's records against the full ones;
more points in a bin than one subproblem takes."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("crowded", [False, True])
@pytest.mark.parametrize("nch", [1, 2, 3, 5, 6, 7, 8, 9, 10, 12, 13, 16, 21, 24])
def test_linear_spread_is_the_transposed_interpolation(pkg, dev, nch, crowded):
    rng = np.random.default_rng(nch)
    L, us, B, Lp = (5, 2, 5, 16) if crowded else (9, 1, 1, 9)
    n = L * us
    pts = rng.uniform(-0.95 * np.pi, 0.95 * np.pi, (B, 3, Lp * Lp))
    if crowded:  # most points within a few cells
        pts[:4] *= 0.05
    pts = torch.tensor(pts.astype(np.float32), device=dev)
    p = pkg.nufft_plan._Plan(L, 27, 1e-6, pkg._lib.KERNEL_LINEAR, us, device=dev)
    p.setpts(pts, wrap=False)
    # the weights: interpolations of the grid's unit vectors, 27 at a time
    eye = torch.eye(n**3, dtype=torch.complex64, device=dev).reshape(-1, n, n, n)
    weights = torch.cat([p.interp(e).real for e in eye.split(27)]).double()  # (n^3, points)
    vals = torch.tensor((rng.standard_normal((nch, pts.shape[0] * Lp * Lp))
                         + 1j * rng.standard_normal((nch, pts.shape[0] * Lp * Lp))).astype(np.complex64), device=dev)
    want = (weights.to(torch.complex128) @ vals.to(torch.complex128).T).T
    out = p.spread(vals).reshape(nch, -1)
    # 32-bit weights (three products) and sums of at most 1280 terms, adding as a random walk: 36 x 6e-8
    assert (out - want).norm() < 2.2e-6 * want.norm()
    # the real part from the records of real volumes, whose indices differ by at most 4.8e-6 cells
    real = p.backproject(vals, None, pkg._lib.REAL_OUTPUT, 1.0).real.double()
    full = p.type1(vals).real.double()
    assert (real - full).norm() < 3**0.5 * 3.1 * 4.8e-6 * full.norm()
