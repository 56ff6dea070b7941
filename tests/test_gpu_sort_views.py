"""A plan's sorted records are those of its current points for every stream, captured or not, from the
first operator on: nothing here warms a view up before it matters."""
import pytest
import torch

pytestmark = pytest.mark.gpu

L, R, B = 16, 3, 64


def _rotations(dev, seed, B=B):
    g = torch.Generator(device=dev).manual_seed(seed)
    q = torch.randn((B, 4), generator=g, device=dev, dtype=torch.float64)
    w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w), 2 * (x * y + z * w),
                        1 - 2 * (x * x + z * z), 2 * (y * z - x * w), 2 * (x * z - y * w), 2 * (y * z + x * w),
                        1 - 2 * (x * x + y * y)], dim=1).reshape(B, 3, 3).float()


def _plan(pkg, kernel, dev):
    return pkg.nufft_plan._Plan(L, R, 1e-6, kernel, 2, width=6 if kernel == 0 else 0, device=dev)


def _grid(p, dev):
    """The native grid of real volumes, made by another plan's transform."""
    g = torch.Generator(device=dev).manual_seed(1)
    return p.fine_grid(torch.randn((R, L, L, L), generator=g, device=dev))


def _outputs(pkg, p, grid):
    return p.interp_native(grid), p.interp_native(grid, None, pkg._lib.GRID_HERMITIAN)


def _want(pkg, kernel, dev, rot, grid):
    p = _plan(pkg, kernel, dev)
    p.setrot(rot, L)
    out = _outputs(pkg, p, grid)
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("kernel", [0, 1])
@pytest.mark.parametrize("hermitian_first", [False, True])
def test_first_operators_on_several_streams(pkg, dev, kernel, hermitian_first):
    """Points set on one stream, the first operators on others that do not wait for one another."""
    grid = _grid(_plan(pkg, kernel, dev), dev)
    rot = _rotations(dev, 2)
    want = _want(pkg, kernel, dev, rot, grid)
    p = _plan(pkg, kernel, dev)
    a, b, c, d = (torch.cuda.Stream() for _ in range(4))
    torch.cuda.synchronize()
    with torch.cuda.stream(a):
        p.setrot(rot, L)
    a.synchronize()
    flags = [pkg._lib.GRID_HERMITIAN if h else 0 for h in (hermitian_first, hermitian_first, not hermitian_first)]
    out = []
    for s, f in zip((b, c, d), flags):
        with torch.cuda.stream(s):
            out.append(p.interp_native(grid, None, f))
    torch.cuda.synchronize()
    for o, f in zip(out, flags):
        assert torch.equal(o, want[1 if f else 0])


@pytest.mark.parametrize("kernel", [0, 1])
@pytest.mark.parametrize("reserved", [False, True])
@pytest.mark.parametrize("hermitian", [False, True])
def test_capture_as_the_first_use(pkg, dev, kernel, reserved, hermitian):
    """The first operator after the points is captured: an eager call before the replay, a second graph
    replayed first, the replay itself and calls after a dropped graph all see the points."""
    grid = _grid(_plan(pkg, kernel, dev), dev)
    rot, rot2 = _rotations(dev, 2), _rotations(dev, 3)
    want, want2 = (_want(pkg, kernel, dev, x, grid) for x in (rot, rot2))
    flags = pkg._lib.GRID_HERMITIAN if hermitian else 0

    def same(out, w):
        # an unreserved plan cannot allocate the pairs' records inside a capture: single records there,
        # whose indices differ by at most 4.8e-6 cells (rounding at n = 32), pi / 2 of the norm each
        torch.cuda.synchronize()
        exact = w[1 if hermitian else 0]
        assert torch.equal(out, exact) or (hermitian and not reserved and torch.equal(out, w[0]))
        assert (out - exact).norm() <= 3**0.5 * 1.6 * 4.8e-6 * exact.norm()

    def captured(p, s):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            out = p.interp_native(grid, None, flags)
        return graph, out

    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        p = _plan(pkg, kernel, dev)
        if reserved:
            p.reserve(B, L, R)
        p.setrot(rot, L)
        graph, _ = captured(p, s)
        del graph  # dropped without a replay
        first, out1 = captured(p, s)
        same(p.interp_native(grid, None, flags), want)
        second, out2 = captured(p, s)
        second.replay()
        same(out2, want)
        first.replay()
        same(out1, want)
        p.setrot(rot2, L)
        first.replay()
        same(out1, want2)
        same(p.interp_native(grid, None, flags), want2)


@pytest.mark.parametrize("kernel", [0, 1])
@pytest.mark.parametrize("hermitian", [False, True])
def test_capture_right_after_the_first_use(pkg, dev, kernel, hermitian):
    """The first operator is launched on one stream and the next one captured on another that does not wait
    for it."""
    grid = _grid(_plan(pkg, kernel, dev), dev)
    rot = _rotations(dev, 2)
    want = _want(pkg, kernel, dev, rot, grid)[1 if hermitian else 0]
    flags = pkg._lib.GRID_HERMITIAN if hermitian else 0
    p = _plan(pkg, kernel, dev)
    a, b, c = (torch.cuda.Stream() for _ in range(3))
    torch.cuda.synchronize()
    with torch.cuda.stream(a):
        p.setrot(rot, L)
    with torch.cuda.stream(b):
        first = p.interp_native(grid, None, flags)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(c):
        graph.capture_begin()
        out = p.interp_native(grid, None, flags)
        graph.capture_end()
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(first, want) and torch.equal(out, want)


@pytest.mark.parametrize("kernel", [0, 1])
@pytest.mark.parametrize("used", ["none", "full"])
def test_points_set_by_a_replay_reach_every_view(pkg, dev, kernel, used):
    """Poses set inside a graph: a plan that has no room for the pairs' records there leaves them out."""
    grid = _grid(_plan(pkg, kernel, dev), dev)
    rots = [_rotations(dev, k) for k in (2, 3, 4)]
    wants = [_want(pkg, kernel, dev, x, grid) for x in rots]
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        p = _plan(pkg, kernel, dev)
        p.setrot(rots[0], L)
        if used == "full":
            p.interp_native(grid)
        static = rots[0].clone()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            p.setrot(static, L)
        for k in (1, 2):
            static.copy_(rots[k])
            graph.replay()
            full, pairs = _outputs(pkg, p, grid)
            torch.cuda.synchronize()
            assert torch.equal(full, wants[k][0])
            assert (pairs - wants[k][1]).norm() <= 3**0.5 * 1.6 * 4.8e-6 * wants[k][1].norm()


def test_points_that_were_refused_leave_none(pkg, dev):
    """A point set past the limit leaves the plan without points, not with stale records."""
    p = _plan(pkg, 1, dev)
    p.setrot(_rotations(dev, 2), L)
    grid = _grid(p, dev)
    p.interp_native(grid)
    with pytest.raises(ValueError):
        pkg._lib.call("cov3d_setrot", p.bind(), pkg._lib.ptr(_rotations(dev, 2)), B, 1 << 14)
    with pytest.raises(RuntimeError):
        p.interp_native(grid)
