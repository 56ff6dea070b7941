"""Mirror-pair records (one per pixels k and -k) against one record per point, over the forms a
plan's points take: the operators on a real volume use the pairs, on the same volume given as
complex (or without the real-output flag) they do not."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# A pair's record may sit 1.5e-7 n <= 1.1e-5 cells from either point (n <= 72); the transform of a
# volume of L voxels changes by at most pi L / n <= 3.1 of its norm per cell and axis
TOL = 3**0.5 * 3.1 * 1.1e-5


def _points(kind, B, L, dev, g):
    q = torch.randn((B, 4), generator=g, device=dev, dtype=torch.float64)
    w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
    R = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w), 2 * (x * y + z * w),
                     1 - 2 * (x * x + z * z), 2 * (y * z - x * w), 2 * (x * z - y * w), 2 * (y * z + x * w),
                     1 - 2 * (x * x + y * y)], dim=1).reshape(B, 3, 3).float()
    if kind == "rot":
        return R, None
    k = torch.ceil(torch.arange(L, device=dev, dtype=torch.float32) - L / 2) / (L / 2) * np.pi
    yy, xx = (t.reshape(-1) for t in torch.meshgrid(k, k, indexing="ij"))
    p = torch.stack([R[:, d, 0, None] * xx + R[:, d, 1, None] * yy for d in (2, 1, 0)], dim=1)
    if kind == "scattered":  # nothing mirrors anything
        p = (torch.rand((B, 3, L * L), generator=g, device=dev) * 2 - 1) * 3.3
    elif kind == "mixed":  # some pairs moved apart, a few by far
        p = p + torch.randn(p.shape, generator=g, device=dev) * 10.0 ** torch.randint(-8, 0, p.shape, device=dev,
                                                                                   generator=g)
    elif kind == "slices":
        p = torch.remainder(p + np.pi, 2 * np.pi) - np.pi
    return None, p.contiguous()


def _plan(pkg, kernel, width, L, us, r, dev):
    return pkg.nufft_plan._Plan(L, r, 1e-6, kernel, us, width=width, device=dev)


@pytest.mark.parametrize("kind", ["rot", "slices", "mixed", "scattered"])
@pytest.mark.parametrize("kernel,width,L,Lp,us,r", [
    (0, 6, 16, 16, 2, 10), (0, 6, 15, 15, 2, 3), (0, 4, 12, 9, 2, 1), (0, 5, 16, 8, 3, 2), (0, 7, 24, 24, 3, 5),
    (0, 8, 13, 13, 3, 4), (1, 0, 16, 16, 2, 10), (1, 0, 15, 15, 1, 4), (1, 0, 16, 11, 1, 1),
    (1, 0, 9, 9, 3, 21)])
def test_pairs_match_single_records(pkg, dev, kind, kernel, width, L, Lp, us, r):
    g = torch.Generator(device=dev).manual_seed(11)
    B = 5
    R, pts = _points(kind, B, Lp, dev, g)
    vol = torch.randn((r, L, L, L), generator=g, device=dev)
    ctf = torch.rand((B, Lp * Lp), generator=g, device=dev) + 0.2
    vals = torch.randn((r, B * Lp * Lp), generator=g, device=dev, dtype=torch.complex64)
    p = _plan(pkg, kernel, width, L, us, r, dev)
    if R is not None:
        p.setrot(R, Lp)
    else:
        p.setpts(pts, wrap=kernel == 0)
    for flags in (0, pkg._lib.APPLY_NYQUIST):
        a = p.project(vol, ctf, flags, 0.5)
        b = p.project(vol.to(torch.complex64), ctf, flags, 0.5)
        assert torch.isfinite(torch.view_as_real(a)).all()
        assert ((a - b).norm() / b.norm()).item() < TOL
        a = p.backproject(vals, ctf, flags | pkg._lib.REAL_OUTPUT, 0.5).real
        b = p.backproject(vals, ctf, flags, 0.5).real
        assert ((a - b).norm() / b.norm()).item() < TOL
    # a new point set reaches both views
    R, pts = _points("rot", B, Lp, dev, g)
    p.setrot(R, Lp)
    a, b = p.project(vol, ctf, 0, 0.5), p.project(vol.to(torch.complex64), ctf, 0, 0.5)
    assert ((a - b).norm() / b.norm()).item() < TOL


def test_pairs_without_upsampling(pkg, dev):
    """At upsampling 1 the deapodised volume's transform is orders above the projections it cancels
    to, so index rounding shows in both forms: the pairs' error against the ES sums in 64 bits is no
    larger than the single records' (up to the scatter of one draw)."""
    from oracle import nufft_oracle as O

    g = torch.Generator(device=dev).manual_seed(11)
    B, L, r = 3, 32, 3
    R, _ = _points("rot", B, L, dev, g)
    vol = torch.randn((r, L, L, L), generator=g, device=dev)
    p = _plan(pkg, 0, 6, L, 1, r, dev)
    p.setrot(R, L)
    want = O.es_type2(vol.cpu().numpy().astype(np.float64), O.rotated_points(R.cpu().numpy().astype(np.float64), L),
                      upsample=1, width=6).reshape(r, -1)
    pair = np.linalg.norm(p.project(vol).cpu().numpy() - want)
    single = np.linalg.norm(p.project(vol.to(torch.complex64)).cpu().numpy() - want)
    assert pair < 1.5 * single


def test_replayed_graph_reads_the_points_set_since(pkg, dev):
    """A step captured after a warm-up reads the poses set before its replay; poses set inside a
    captured graph reach a later call outside it, whichever records that call uses."""
    L, r, B = 16, 2, 6
    g = torch.Generator(device=dev).manual_seed(3)
    rot = [_points("rot", B, L, dev, g)[0] for _ in range(3)]
    vol = torch.randn((r, L, L, L), generator=g, device=dev)
    p, ref = _plan(pkg, 0, 6, L, 2, r, dev), _plan(pkg, 0, 6, L, 2, r, dev)

    def want(R, complex_volume):
        ref.setrot(R, L)
        return ref.project(vol.to(torch.complex64) if complex_volume else vol)

    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        p.setrot(rot[0], L)
        p.project(vol)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            out = p.project(vol)
        p.setrot(rot[1], L)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want(rot[1], False))
        static = rot[0].clone()
        points = torch.cuda.CUDAGraph()
        with torch.cuda.graph(points, stream=s):
            p.setrot(static, L)
        static.copy_(rot[2])
        points.replay()
        torch.cuda.synchronize()
        assert torch.equal(p.project(vol), want(rot[2], False))
        full = p.project(vol.to(torch.complex64))
        static.copy_(rot[1])
        points.replay()
        torch.cuda.synchronize()
        assert torch.equal(full, want(rot[2], True))
        assert torch.equal(p.project(vol.to(torch.complex64)), want(rot[1], True))
