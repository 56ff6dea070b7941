"""ES interpolation with units of points sharing a tile load (dense bins) and point by point (sparse
bins): the same points give the same bits whichever kernel their number selects, so a batch is compared
with its images one at a time, and with the 64-bit ES sums."""
import numpy as np
import pytest
import torch

from oracle import nufft_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["rot", "crowded"])
@pytest.mark.parametrize("width,r,L", [(4, 10, 16), (4, 3, 9), (5, 12, 12), (5, 1, 11), (6, 10, 16), (6, 20, 12),
                                       (6, 13, 10), (6, 6, 11), (6, 5, 16), (6, 3, 13), (6, 2, 8), (6, 1, 16),
                                       (7, 10, 16), (7, 7, 10), (7, 4, 11), (7, 2, 20)])
def test_dense_batch_has_the_bits_of_single_images(pkg, dev, width, r, L, kind):
    g = torch.Generator(device=dev).manual_seed(width * 31 + r)
    B = 12 * L  # three points per cell and more
    vol = torch.randn((r, L, L, L), generator=g, device=dev)
    ctf = torch.rand((B, L * L), generator=g, device=dev) + 0.2
    p = pkg.nufft_plan._Plan(L, r, 1e-6, pkg._lib.KERNEL_ES, 2, width=width, device=dev)
    if kind == "rot":
        poses = torch.linalg.qr(torch.randn((B, 3, 3), device=dev, generator=g))[0].contiguous()
        put = lambda i, j: p.setrot(poses[i:j].contiguous(), L)  # noqa: E731
    else:
        poses = (torch.rand((B, 3, L * L), generator=g, device=dev) * 2 - 1) * 0.3
        put = lambda i, j: p.setpts(poses[i:j].contiguous(), wrap=True)  # noqa: E731
    for v in (vol, vol.to(torch.complex64)):  # mirror pairs, one record per point
        put(0, B)
        whole = p.project(v, ctf, pkg._lib.APPLY_NYQUIST, 0.5).reshape(r, B, -1)
        for i in (0, B // 2, B - 1):
            put(i, i + 1)
            assert torch.equal(p.project(v, ctf[i:i + 1].contiguous(), pkg._lib.APPLY_NYQUIST, 0.5), whole[:, i])
    if kind == "crowded":
        put(0, 2)
        got = p.type2(vol).reshape(r, 2, -1).cpu().numpy()
        put(0, B)
        assert np.array_equal(p.type2(vol).reshape(r, B, -1)[:, :2].cpu().numpy(), got)
        want = O.es_type2(vol.cpu().numpy().astype(np.float64), poses[:2].cpu().numpy().astype(np.float64), upsample=2,
                          width=width)
        # weights to 1e-6 (fast exponential), indices to 1.2e-7 n cells at a slope of pi / 2 per cell and axis
        assert np.linalg.norm(got - want) < (3e-6 + 3**0.5 * 1.6 * 1.2e-7 * 2 * L) * np.linalg.norm(want)
