"""Per-image solves against numpy at the ranks where the kernel's classes and images per block change,
with batches that end within a block, and one matrix that is not positive definite."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r,B", [(1, 65), (9, 13), (10, 12), (11, 1), (16, 8), (17, 9), (20, 7), (21, 6), (32, 4)])
@pytest.mark.parametrize("objective", [0, 1])
def test_solve_matches_numpy(pkg, dev, r, B, objective):
    rng = np.random.default_rng(r)
    A = (rng.standard_normal((B, r, 2 * r)) + 1j * rng.standard_normal((B, r, 2 * r))).astype(np.complex64)
    gram = (A @ A.conj().transpose(0, 2, 1)).astype(np.complex64)
    gram = (0.5 * (gram + gram.conj().transpose(0, 2, 1))).astype(np.complex64)
    h = (rng.standard_normal((B, r)) + 1j * rng.standard_normal((B, r))).astype(np.complex64)
    broken = B // 2 if objective == 0 and B > 4 else None
    if broken is not None:
        gram[broken, r - 1, r - 1] = -1e4
    s2 = 1.5
    t = lambda v: torch.tensor(v, device=dev)  # noqa: E731
    out = dict(C=(B, r, r), u=(B, r), z=(B, r), m=(B, r, r))
    out = {k: torch.zeros(s, dtype=torch.complex64, device=dev) for k, s in out.items()}
    cost = torch.zeros(B, dtype=torch.float64, device=dev)
    bad = torch.zeros(1, dtype=torch.int32, device=dev)
    G, H, ptr = t(gram), t(h), pkg._lib.ptr
    pkg._lib.call("cov3d_cost_solve", pkg._lib.stream_ptr(dev), B, r, objective, ptr(G), ptr(H), s2, None, 0.5, 1.0,
                  ptr(out["C"]), ptr(out["u"]), ptr(cost), None, ptr(out["z"]), ptr(out["m"]), ptr(bad))
    assert int(bad.item()) == (broken is not None)
    g, hh = gram.astype(np.complex128), h.astype(np.complex128)
    keep = [b for b in range(B) if b != broken]
    if objective == 0:
        m = g / s2 + np.eye(r)
        b = hh / s2
        z = np.linalg.solve(m, b[..., None])[..., 0]
        minv = np.linalg.inv(m)
        want = dict(m=m, z=z, u=-z.conj() / (4 * s2),
                    C=(minv.conj() + z.conj()[:, :, None] * z[:, None, :]) / (4 * s2))
        cw = 0.5 * (-(b.conj() * z).sum(1).real + np.linalg.slogdet(m)[1])
    else:
        want = dict(u=-hh.conj(), C=0.5 * (2 * g.conj() + 2 * s2 * np.eye(r)))
        h2 = (abs(hh) ** 2).sum(1)
        cw = -2 * h2 + (abs(g) ** 2).sum((1, 2)) + 2 * s2 * np.trace(g, axis1=1, axis2=2).real
    for k, w in want.items():
        w = w[keep]
        # outputs round once to 32 bits (6e-8); 64-bit solves of matrices conditioned below 1e3 add 1e-12
        assert abs(out[k].cpu().numpy()[keep] - w).max() < 2e-7 * abs(w).max(), k
    assert abs(cost.cpu().numpy()[keep] - cw[keep]).max() < 1e-11 * abs(cw[keep]).max()
