"""Nearest-cell spreading at the channel counts where its launches change (pairs of channels, one to five
of them, then another launch), point-major and channel-major, against 64-bit sums; more points in a bin
than a chunk of the kernel and than a block takes."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("crowded", [False, True])
@pytest.mark.parametrize("point_major", [False, True])
@pytest.mark.parametrize("nch", [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 20, 21])
def test_channel_counts(pkg, dev, nch, point_major, crowded):
    rng = np.random.default_rng(nch)
    n, us, B, Lp = 22, 2, (40 if crowded else 3), 14
    M = B * Lp * Lp
    cell = rng.integers(0, n, (M, 3))
    if crowded:  # most points in the eight cells of one bin's corner
        cell[: 9 * M // 10] = rng.integers(0, 2, (9 * M // 10, 3)) + 1
    w = (cell - n // 2 + rng.uniform(-0.2, 0.2, cell.shape)) * (2 * np.pi / n)
    pts = np.ascontiguousarray(w.reshape(B, Lp * Lp, 3).transpose(0, 2, 1).astype(np.float32))
    vals = (rng.standard_normal((nch, M)) + 1j * rng.standard_normal((nch, M))).astype(np.complex64)
    p = pkg.nufft_plan._Plan(n // us, nch, 1e-6, pkg._lib.KERNEL_NEAREST, us, device=dev)
    p.setpts(torch.tensor(pts, device=dev), wrap=False)
    want = np.zeros((nch, n, n, n), np.complex128)
    for c in range(nch):
        np.add.at(want[c], tuple(cell.T), vals[c].astype(np.complex128))
    lay = pkg._lib.GridLayout(order=pkg._lib.GRID_CENTERED, cell_stride=1, chan_stride=n**3)
    grid = torch.zeros((nch, n, n, n), dtype=torch.complex64, device=dev)
    v = torch.tensor(np.ascontiguousarray(vals.T) if point_major else vals, device=dev)
    strides = (nch, 1) if point_major else (1, M)
    pkg._lib.call("cov3d_spread", p.bind(), pkg._lib.ptr(v), *strides, nch, None, 0, 1.0, pkg._lib.ptr(grid),
                  pkg._lib.ctypes.byref(lay), 1)
    # TwoSum sums round once per block and cell (at most three blocks meet in a cell here)
    assert np.linalg.norm(grid.cpu().numpy() - want) < 2e-7 * np.linalg.norm(want)
