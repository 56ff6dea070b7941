"""Per-image Gram and its adjoint's W = C Q + u y against 64-bit sums, at the ranks where tiles, pixel groups
and register classes change, with images that end within a chunk, point-major, channel-major and padded."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r,P,B", [(1, 1, 3), (2, 127, 2), (3, 128, 2), (4, 129, 3), (5, 1025, 2), (8, 900, 3),
                                   (9, 2000, 2), (14, 300, 2), (15, 300, 2), (20, 1100, 3), (21, 257, 1), (22, 513, 2),
                                   (32, 700, 2)])
@pytest.mark.parametrize("layout", ["point", "channel", "padded"])
def test_gram_and_wpass_match_64_bit_sums(pkg, dev, r, P, B, layout):
    rng = np.random.default_rng(r + P)
    rnd = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)  # noqa: E731
    q, y, C, u = rnd(B, r, P), rnd(B, P), rnd(B, r, r), rnd(B, r)
    if layout == "channel":
        store, (si, sp, sc) = q, (r * P, 1, P)
    elif layout == "point":
        store, (si, sp, sc) = q.transpose(0, 2, 1), (r * P, r, 1)
    else:  # point-major rows of r + 3, images padded
        store, (si, sp, sc) = np.zeros((B, P + 1, r + 3), np.complex64), ((P + 1) * (r + 3), r + 3, 1)
        store[:, :P, :r] = q.transpose(0, 2, 1)
    t = lambda v: torch.tensor(np.ascontiguousarray(v), device=dev)  # noqa: E731
    Q, Y, Cd, ud, ptr = t(store), t(y), t(C), t(u), pkg._lib.ptr
    gram = torch.zeros((B, r, r), dtype=torch.complex64, device=dev)
    h = torch.zeros((B, r), dtype=torch.complex64, device=dev)
    yy = torch.zeros((B,), dtype=torch.float32, device=dev)
    st = pkg._lib.stream_ptr(dev)
    pkg._lib.call("cov3d_gram", st, B, P, r, ptr(Q), si, sp, sc, ptr(Y), ptr(gram), ptr(h), ptr(yy))
    v = np.concatenate([q, y[:, None]], 1).astype(np.complex128)
    want = v.conj() @ v.transpose(0, 2, 1)
    got = want.copy()
    got[:, :r, :r], got[:, :r, r], got[:, r, r] = gram.cpu().numpy(), h.cpu().numpy(), yy.cpu().numpy()
    norm = np.sqrt(np.einsum("bii->bi", want).real)
    # chains of up to 128 pixels, two roundings each, then compensated: 256 x 6e-8 of the factors' norms
    assert (abs(got - want)[:, :, r] <= 1.6e-5 * norm * norm[:, r:]).all()
    assert (abs(got - want)[:, :r, :r] <= 1.6e-5 * norm[:, :r, None] * norm[:, None, :r]).all()
    assert np.linalg.norm(got - want) < 1e-6 * np.linalg.norm(want)
    W = torch.zeros_like(Q)
    for out in (W, Q):  # beside Q, then over it
        pkg._lib.call("cov3d_wpass", st, B, P, r, ptr(Q), si, sp, sc, ptr(Y), ptr(Cd), ptr(ud), ptr(out), si, sp, sc)
        res = out.cpu().numpy()
        res = res if layout == "channel" else res[:, :P, :r].transpose(0, 2, 1)
        wantw = C.astype(np.complex128) @ v[:, :r] + u[:, :, None].astype(np.complex128) * v[:, r:]
        # r + 1 terms of four products: at most 66 roundings of 6e-8, adding as a random walk
        assert np.linalg.norm(res - wantw) < 1e-6 * np.linalg.norm(wantw)
