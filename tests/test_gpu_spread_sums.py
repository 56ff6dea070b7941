"""Summation accuracy of the spreading where many points meet in a cell: central slices of many images
all pass through the origin.  The reference is the 64-bit sum of the spreadings of the single images,
which have the same weights to the bit, so only the order and precision of the sums differ."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rotations(dev, B, seed):
    g = torch.Generator(device=dev).manual_seed(seed)
    q = torch.randn((B, 4), generator=g, device=dev, dtype=torch.float64)
    w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w), 2 * (x * y + z * w),
                        1 - 2 * (x * x + z * z), 2 * (y * z - x * w), 2 * (x * z - y * w), 2 * (y * z + x * w),
                        1 - 2 * (x * x + y * y)], dim=1).reshape(B, 3, 3).float()


# Relative errors of the compensated row sums (two or three FP32 sums per subproblem folded by TwoSum,
# one atomic addition per cell and subproblem) on these very inputs, the largest of four runs: the 9^3 cells
# around the origin and all cells, values of one sign and of both.  The sums here may be no further off,
# up to the scatter from run to run (a fifth near the origin, a tenth over all cells).
ROW_SUMS = {
    (0, 4, 2, 10): ((1.40e-7, 0.90e-7), (1.77e-7, 1.28e-7)), (0, 5, 2, 5): ((1.11e-7, 0.89e-7), (2.01e-7, 1.50e-7)),
    (0, 6, 2, 1): ((1.58e-7, 1.09e-7), (2.11e-7, 1.68e-7)), (0, 6, 2, 2): ((1.50e-7, 1.07e-7), (2.22e-7, 1.68e-7)),
    (0, 6, 2, 4): ((1.45e-7, 1.06e-7), (2.21e-7, 1.68e-7)), (0, 6, 2, 5): ((1.17e-7, 1.00e-7), (2.21e-7, 1.76e-7)),
    (0, 6, 2, 10): ((1.22e-7, 1.01e-7), (2.17e-7, 1.76e-7)), (0, 7, 2, 1): ((1.60e-7, 1.19e-7), (2.48e-7, 1.99e-7)),
    (0, 7, 2, 10): ((1.24e-7, 1.09e-7), (2.43e-7, 1.99e-7)), (0, 8, 2, 1): ((1.50e-7, 1.26e-7), (2.55e-7, 2.13e-7)),
    (1, 0, 2, 1): ((0.84e-7, 0.65e-7), (1.00e-7, 0.77e-7)), (1, 0, 2, 2): ((0.84e-7, 0.65e-7), (1.28e-7, 0.79e-7)),
    (1, 0, 1, 2): ((1.57e-7, 1.24e-7), (2.20e-7, 1.50e-7)), (1, 0, 2, 3): ((0.92e-7, 0.68e-7), (1.14e-7, 0.78e-7)),
    (1, 0, 2, 5): ((0.92e-7, 0.68e-7), (1.14e-7, 0.77e-7)), (1, 0, 2, 8): ((0.92e-7, 0.68e-7), (1.14e-7, 0.77e-7)),
    (1, 0, 2, 10): ((0.92e-7, 0.68e-7), (1.14e-7, 0.77e-7)), (2, 0, 2, 2): ((0.84e-7, 0.57e-7), (0.75e-7, 0.46e-7)),
    (2, 0, 2, 10): ((0.84e-7, 0.57e-7), (0.77e-7, 0.47e-7)),
}


@pytest.mark.parametrize("signs", [0, 1])
@pytest.mark.parametrize("kernel,width,us,nch", list(ROW_SUMS))
def test_crowded_cells(pkg, dev, kernel, width, us, nch, signs):
    L, B = 24, 600
    R = _rotations(dev, B, 5)
    g = torch.Generator(device=dev).manual_seed(7)
    v = torch.randn((nch, B, L * L), generator=g, device=dev, dtype=torch.complex64)
    if signs == 0:
        v = (1.0 + 0.3 * v.abs()).to(torch.complex64)
    p, q = (pkg.nufft_plan._Plan(L, nch, 1e-6, kernel, us, width=width, device=dev) for _ in range(2))
    p.setrot(R, L)
    got = p.spread(v.reshape(nch, -1))
    want = torch.zeros(got.shape, dtype=torch.complex128, device=dev)
    for b in range(B):
        q.setrot(R[b:b + 1].contiguous(), L)
        want += q.spread(v[:, b].contiguous())
    c, k = p.n // 2, 4
    box = (slice(None),) + (slice(c - k, c + k + 1),) * 3
    near, whole = ROW_SUMS[kernel, width, us, nch][signs]
    assert (got[box] - want[box]).norm() < 1.2 * near * want[box].norm()
    assert (got - want).norm() < 1.1 * whole * want.norm()
