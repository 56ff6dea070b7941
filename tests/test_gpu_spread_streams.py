"""Accumulating calls of two plans on two streams onto one grid lose nothing."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel,width,nch", [(2, 0, 1), (2, 0, 2), (2, 0, 5), (1, 0, 2), (0, 6, 2)])
def test_two_streams_add_to_one_grid(pkg, dev, kernel, width, nch):
    L, B = 32, 96
    lib = pkg._lib
    g = torch.Generator(device=dev).manual_seed(3)
    pts = (torch.rand((B, 3, L * L), generator=g, device=dev) * 2 - 1) * 3.0
    # whole numbers (their sums are exact in any order where the weights are)
    vals = torch.randint(-8, 9, (nch, B * L * L), generator=g, device=dev).to(torch.complex64)
    plans = [pkg.nufft_plan._Plan(L, nch, 1e-6, kernel, 2, width=width, device=dev) for _ in range(2)]
    for p in plans:
        p.setpts(pts, wrap=kernel == 0)
        one = p.spread(vals)
    n = plans[0].n
    grid = torch.zeros_like(one)
    layout = lib.GridLayout(order=lib.GRID_CENTERED, cell_stride=1, chan_stride=n**3)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for _ in range(4):
        for p, s in zip(plans, streams):
            with torch.cuda.stream(s):
                lib.call("cov3d_spread", p.bind(), lib.ptr(vals), 1, p.n_points, nch, None, 0, 1.0, lib.ptr(grid),
                         lib.ctypes.byref(layout), 1)
    torch.cuda.synchronize()
    if kernel == 2:
        assert torch.equal(grid, 8 * one)
    else:  # 8 x the sum of at most some hundred terms per cell in FP32
        assert (grid - 8 * one).norm() < 1e-5 * grid.norm()
