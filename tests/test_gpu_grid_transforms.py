"""The plans' volume <-> fine grid transforms against 64-bit FFTs: each line-kernel size, batched small
grids, grids above them with even and odd volumes, real and complex volumes."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# n = 64, 128, 256, 512 (line kernels; cuFFT forward at 512), 60, 62 (batched), 162, 176 (per channel, odd L
# and even L), a volume no larger than a quarter of the grid, an L that is no multiple of four
@pytest.mark.parametrize("L,us,C", [(32, 2, 3), (64, 2, 2), (16, 8, 2), (128, 2, 1), (128, 4, 1), (30, 2, 5), (31, 2, 2),
                                    (81, 2, 2), (88, 2, 2), (33, 5, 1), (4, 16, 2), (24, 1, 2)])
@pytest.mark.parametrize("real", [True, False])
def test_grid_transforms_match_64_bit_ffts(pkg, dev, L, us, C, real):
    rng = np.random.default_rng(L + us)
    n = L * us
    p = pkg.nufft_plan._Plan(L, C, 1e-6, pkg._lib.KERNEL_LINEAR, us, device=dev)
    gc = p.grid_correction().cpu().numpy().astype(np.float64).reshape(L, L, L)
    v = rng.standard_normal((C, L, L, L)).astype(np.float32)
    if not real:
        v = (v + 1j * rng.standard_normal(v.shape)).astype(np.complex64)
    ax = (np.arange(L) - L // 2) % n
    box = (slice(None),) + np.ix_(ax, ax, ax)
    want = np.zeros((C, n, n, n), np.complex128)
    want[box] = v / gc
    want = np.fft.fftn(want, axes=(1, 2, 3))
    grid = p.fine_grid(torch.tensor(v, device=dev)).cpu().numpy().reshape(C, n, n, n)
    # three passes of 32-bit butterflies of at most log2(n) = 9 levels: 27 roundings of 6e-8 add to 3e-7
    assert np.linalg.norm(grid - want) < 1e-6 * np.linalg.norm(want)

    Lp = min(L, 32)
    pts = rng.uniform(-np.pi, np.pi, (2, 3, Lp * Lp)).astype(np.float32) * 0.9
    p.setpts(torch.tensor(pts, device=dev), wrap=False)
    vals = (rng.standard_normal((C, 2 * Lp * Lp)) + 1j * rng.standard_normal((C, 2 * Lp * Lp))).astype(np.complex64)
    spread = p.spread(torch.tensor(vals, device=dev)).cpu().numpy().reshape(C, n, n, n).astype(np.complex128)
    back = np.fft.ifftn(np.fft.ifftshift(spread, axes=(1, 2, 3)), axes=(1, 2, 3), norm="forward")[box] / gc
    out = p.type1(torch.tensor(vals, device=dev)).cpu().numpy().reshape(back.shape)
    assert np.linalg.norm(out - back) < 1e-6 * np.linalg.norm(back)
