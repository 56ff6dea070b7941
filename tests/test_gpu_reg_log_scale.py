"""The regulariser's derivative with respect to log_sqrt where its terms differ by 24 bits: one row of
cells in sixteen holds the sum, the others a part in a million of it that FP32 sums would drop."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_channel", [False, True])
def test_small_terms_next_to_large_ones(pkg, dev, per_channel):
    L, r = 100, 2
    n = 2 * L
    g = torch.Generator(device=dev).manual_seed(1)
    vec = torch.randn((r, L, L, L), generator=g, device=dev) / L**1.5
    step = pkg.FusedCovarStep(L, r, "bilinear", 2, device=dev)
    step.set_rotations(torch.eye(3, device=dev).reshape(1, 3, 3))
    # the first 2432 rows of cells (a capped grid's blocks) in storage order, then the others, far smaller
    fr = torch.full((n * n, n), 5e-8, device=dev)
    fr[:2432] = 1.0
    fr = torch.roll(fr.reshape(n, n, n), (n // 2,) * 3, (0, 1, 2)).contiguous()
    if per_channel:
        fr = torch.stack([fr] * r).contiguous()
    s2 = 1e12  # the data's part vanishes
    _, _, gl = step(vec, torch.zeros(r, device=dev), torch.zeros((1, L * L), dtype=torch.complex64, device=dev), None,
                    s2, 2 * s2, fr, 0)
    v = vec.double() / step.plan.grid_correction().double()
    pad = torch.zeros((r, n, n, n), dtype=torch.float64, device=dev)
    o = n // 2 - L // 2
    pad[:, o:o + L, o:o + L, o:o + L] = v
    G = torch.fft.fftshift(torch.fft.fftn(torch.fft.ifftshift(pad, dim=(1, 2, 3)), dim=(1, 2, 3)), dim=(1, 2, 3))
    want = 2 * (fr.double() * G.abs() ** 2).reshape(r, -1).sum(1)
    # output rounding 6e-8; the transforms' and weights' rounding averages out over the cells
    assert ((gl.double() - want).abs() < 2e-7 * want).all()
