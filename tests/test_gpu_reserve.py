"""What cov3d_plan_reserve holds: one sorted view of the points for nearest cells, which have no mirror
pairs, and two for the other windows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel,views", [(2, 1), (1, 2), (0, 2)])
def test_reserved_views(pkg, dev, kernel, views):
    p = pkg.nufft_plan._Plan(8, 1, 1e-6, kernel, 2, width=6 if kernel == 0 else 0, device=dev)
    images, L = 16, 512
    M = images * L * L
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info(dev)[0]
    p.reserve(images, L, 1)
    held = before - torch.cuda.mem_get_info(dev)[0]
    # 24 bytes per point and view (record, bin, rank) and the projections' 8, some MB of tables and rounding
    assert abs(held - M * (24 * views + 8)) < 24e6
    g = torch.Generator(device=dev).manual_seed(1)
    pts = (torch.rand((images, 3, L * L), generator=g, device=dev) * 2 - 1) * 3.0
    p.reserve(images, L, 1, points=True)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info(dev)[0]
    p.setpts(pts, wrap=kernel == 0)  # nothing is allocated within the reserved sizes
    assert torch.cuda.mem_get_info(dev)[0] == before
