"""The ES spreading kernel against the 64-bit ES sums: every window width, the channel counts at the
edges of its layouts (passes of ten, five, two, one), grids that are no multiple of the bins, one
image, and more points in a bin than one subproblem takes."""
import numpy as np
import pytest
import torch

from oracle import nufft_oracle as O

pytestmark = pytest.mark.gpu

# float32 indices are good to 1.2e-7 n (the angle's and the index's rounding, n <= 40) = 4.8e-6 cells,
# and the adjoint changes by at most pi / upsampling per cell and axis
TOL = 3**0.5 * 3.1 * 4.8e-6


@pytest.mark.parametrize("crowded", [False, True])
@pytest.mark.parametrize("width,nch,L,us", [
    (4, 1, 9, 2), (4, 10, 16, 2), (5, 2, 11, 2), (5, 6, 12, 2), (6, 1, 16, 2), (6, 2, 13, 3), (6, 3, 16, 2),
    (6, 5, 9, 2), (6, 6, 10, 2), (6, 10, 16, 2), (6, 11, 10, 2), (6, 12, 10, 2), (6, 13, 10, 2), (6, 16, 10, 2),
    (6, 20, 16, 2), (7, 1, 20, 2), (7, 2, 10, 2), (7, 4, 10, 2), (7, 10, 12, 2), (8, 1, 12, 2), (8, 7, 10, 3)])
def test_spread_matches_64_bit_sums(pkg, dev, width, nch, L, us, crowded):
    rng = np.random.default_rng(width * 100 + nch)
    B, Lp = (4, 16) if crowded else (1, 11)
    pts = rng.uniform(-np.pi, np.pi, (B, 3, Lp * Lp))
    if crowded:  # most points within a few cells, across the periodic edge on one axis
        pts[:3] *= 0.05
        pts[0, 1] = np.mod(pts[0, 1] + 2 * np.pi, 2 * np.pi) - np.pi
    pts = pts.astype(np.float32)
    vals = rng.standard_normal((nch, B * Lp * Lp)) + 1j * rng.standard_normal((nch, B * Lp * Lp))
    vals = vals.astype(np.complex64)
    p = pkg.nufft_plan._Plan(L, nch, 1e-6, pkg._lib.KERNEL_ES, us, width=width, device=dev)
    p.setpts(torch.tensor(pts, device=dev), wrap=True)
    want = O.es_type1(vals.astype(np.complex128).reshape(nch, B, -1), pts.astype(np.float64), L, upsample=us, width=width)
    want = want.reshape(nch, L, L, L)
    out = p.type1(torch.tensor(vals, device=dev)).cpu().numpy()
    assert np.linalg.norm(out - want) < TOL * np.linalg.norm(want)
    out = p.backproject(torch.tensor(vals, device=dev), None, pkg._lib.REAL_OUTPUT, 1.0).cpu().numpy().real
    assert np.linalg.norm(out - want.real) < TOL * np.linalg.norm(want.real)
