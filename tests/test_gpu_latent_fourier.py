"""Latent coordinates from Fourier-domain inner products against those from spatial projections: even and
odd images, filters that are not even in the frequency, real and complex images, ragged batches."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,r,n", [(16, 1, 5), (17, 4, 9), (24, 10, 12), (33, 11, 7), (32, 20, 6)])
@pytest.mark.parametrize("cplx", [False, True])
def test_latent_map_equals_spatial_inner_products(pkg, dev, L, r, n, cplx):
    g = torch.Generator(device=dev).manual_seed(L)
    rand = lambda *s: torch.randn(s, device=dev, generator=g)  # noqa: E731
    vols, R = rand(r, L, L, L), torch.linalg.qr(rand(n, 3, 3))[0].contiguous()
    filters, images, lam = rand(n, L, L), rand(n, L, L), rand(r).abs() + 0.5
    if cplx:
        images = torch.complex(images, rand(n, L, L))

    class Data:
        noise_var = 3.0

        def __len__(self):
            return n

        def __getitem__(self, s):
            return images[s], R[s], filters[s], torch.arange(n)[s]

    z, m = pkg.wiener_coords.latentMAP(Data(), vols, lam, batch_size=4, return_coords_covar=True)
    plan = pkg.NufftPlan((L,) * 3, batch_size=r, device=dev)
    plan.setrot(R)
    q = pkg.vol_forward(vols, plan, filters).reshape(n, r, -1).double()
    y = images.reshape(n, -1, 1).to(torch.complex128)
    gram = q @ q.transpose(1, 2) / 3.0
    want_m = gram + torch.diag(1.0 / (lam.double() + 1e-6))
    want = torch.linalg.solve(want_m.to(torch.complex128), q.to(torch.complex128) @ y / 3.0).squeeze(-1).real
    # 32-bit projections (3e-6 between the plans' sums) through well-conditioned matrices
    assert (m.double().to(dev) - want_m).norm() < 1e-5 * want_m.norm()
    cond = torch.linalg.cond(want_m).max().item()
    assert (z.double() - want).norm() < 1e-5 * cond * want.norm()
