"""Nearest-cell spreading against 64-bit sums: grids that are no multiple of the bins, one to three
channels, strided channels, more points in a bin than one block takes, accumulation onto a grid."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,us,B,Lp,nch,crowded", [(10, 1, 1, 5, 1, False), (24, 2, 3, 12, 2, False),
                                                   (16, 2, 5, 16, 3, False), (33, 3, 2, 17, 1, False),
                                                   (16, 2, 90, 16, 2, True), (20, 1, 40, 20, 1, True)])
@pytest.mark.parametrize("compensated", [True, False])
def test_nearest_spread_matches_64_bit_sums(pkg, dev, n, us, B, Lp, nch, crowded, compensated):
    rng = np.random.default_rng(n + nch)
    M = B * Lp * Lp
    cell = rng.integers(0, n, (M, 3))
    if crowded:  # most points in the eight cells of one bin's corner
        cell[: 9 * M // 10] = rng.integers(0, 2, (9 * M // 10, 3)) + 1
    # frequencies a fifth of a cell around the cells' centres: no rounding decides the cell
    w = (cell - n // 2 + rng.uniform(-0.2, 0.2, cell.shape)) * (2 * np.pi / n)
    pts = w.reshape(B, Lp * Lp, 3).transpose(0, 2, 1).astype(np.float32)
    vals = (rng.standard_normal((nch, M)) + 1j * rng.standard_normal((nch, M))).astype(np.complex64)
    p = pkg.nufft_plan._Plan(n // us, nch, 1e-6, pkg._lib.KERNEL_NEAREST, us, compensated=compensated, device=dev)
    p.setpts(torch.tensor(np.ascontiguousarray(pts), device=dev), wrap=False)
    want = np.zeros((nch, n, n, n), np.complex128)
    for c in range(nch):
        np.add.at(want[c], tuple(cell.T), vals[c].astype(np.complex128))
    # TwoSum sums round once per block and cell; plain ones once per point (at most 20736 in a cell)
    tol = 2e-7 if compensated else 6e-8 * np.sqrt(M)
    out = p.spread(torch.tensor(vals, device=dev))
    assert np.linalg.norm(out.cpu().numpy() - want) < tol * np.linalg.norm(want)
    lay = pkg._lib.GridLayout(order=pkg._lib.GRID_CENTERED, cell_stride=nch, chan_stride=1)
    grid = torch.ones((n, n, n, nch), dtype=torch.complex64, device=dev)
    v = torch.tensor(np.ascontiguousarray(vals.T), device=dev)
    pkg._lib.call("cov3d_spread", p.bind(), pkg._lib.ptr(v), nch, 1, nch, None, 0, 1.0, pkg._lib.ptr(grid),
                  pkg._lib.ctypes.byref(lay), 1)
    assert np.linalg.norm(grid.cpu().numpy() - (want.transpose(1, 2, 3, 0) + 1)) < (tol + 2e-7) * np.linalg.norm(want) + \
        6e-8 * np.sqrt(grid.numel())
