"""The work this framework is timed on: its public calls at the sizes they are used at.

Every case is a plain dict; ``prepare`` makes what a program has in hand before the call (inputs
on the GPU from the seed, plans sized once), ``run`` is one pass through the public entry point,
``work`` the bytes and operations that pass cannot do without, and ``exact`` the same result in 64
bits from plain torch.  Volumes are smooth random shapes in a ball, images are noise-dominated
(as cryo-EM images are), poses are uniform on SO(3) unless a case says otherwise.
"""

import importlib
import math

import torch

cov3d = importlib.import_module("3dcovarestimation_gb300")

DEV = torch.device("cuda")
UPSAMPLE = 2


def listed():
    return [
        # one SGD batch of the smallest configuration (2 000 images of 32^2, rank 5), bilinear
        # plans: launches and latency count
        dict(name="step_bilinear_small", kind="step", disc="bilinear", width=0, L=32, r=5, B=256, objective="ml",
             reg=False, ctf="array", poses="rot"),
        # one SGD batch with the command line's default interpolation
        dict(name="step_bilinear", kind="step", disc="bilinear", width=0, L=128, r=10, B=1024, objective="ml",
             reg=True, ctf="array", poses="rot"),
        # the headline: one SGD batch on the exact NUFFT, CTFs evaluated in the kernels
        dict(name="step_nufft", kind="step", disc="nufft", width=6, L=128, r=10, B=1024, objective="ml", reg=True,
             ctf="params", poses="rot"),
        # the same at rank 20, a ragged last batch
        dict(name="step_nufft_r20", kind="step", disc="nufft", width=6, L=128, r=20, B=300, objective="ml", reg=True,
             ctf="params", poses="rot"),
        # the least-squares objective with its regulariser, points given as the reference's pts_rot
        dict(name="step_ls_points", kind="step", disc="nufft", width=6, L=64, r=5, B=500, objective="ls", reg=True,
             ctf="array", poses="pts"),
        # the drop-in cost function under autograd: forward and backward through grid_sample plans
        dict(name="cost_autograd", kind="autograd", L=64, r=8, B=512),
        # projections of a few volumes on the exact plan, odd image size, default tolerance
        dict(name="project_odd", kind="project", L=95, r=4, B=100),
        # backprojection of one batch of images to a volume on the exact plan
        dict(name="backproject", kind="backproject", L=128, B=512),
        # one batch of the mean's backprojection (nearest plan; offsets and contrasts)
        dict(name="mean_add", kind="mean_add", L=128, B=1024),
        # the mean's padding solve: plain conjugate gradients
        dict(name="mean_cg", kind="cg", L=128, precond="none", iters=32),
        # the same with the circulant preconditioner, at a smaller volume
        dict(name="mean_cg_circulant", kind="cg", L=64, precond="circulant", iters=12),
        # Wiener coordinates of a dataset in batches with a ragged last one
        dict(name="latent_map", kind="latent", L=128, r=10, B=1500, batch=1024),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "autograd", "project", "backproject", "mean_add", "cg", "latent"])
    if kind == "step":
        disc = rng.choice(["nufft", "nufft", "bilinear"])
        L = _log_int(rng, 24, 128)
        r = rng.randint(1, 20)
        objective = rng.choice(["ml", "ml", "ml", "ls"]) if L <= 64 else "ml"
        B = min(_log_int(rng, 16, 1024), max(1, 1024 * 128**2 * 10 // (L * L * max(r, 10))))
        return dict(kind=kind, disc=disc, width=rng.choice([5, 6, 6]) if disc == "nufft" else 0, L=L, r=r, B=B,
                    objective=objective, reg=rng.random() < 0.7, ctf=rng.choice(["array", "params"]),
                    poses=rng.choice(["rot", "rot", "pts"]))
    if kind == "autograd":
        L = _log_int(rng, 20, 80)
        return dict(kind=kind, L=L, r=rng.randint(1, 12), B=_log_int(rng, 16, 512))
    if kind == "project":
        return dict(kind=kind, L=_log_int(rng, 24, 128), r=rng.randint(1, 10), B=_log_int(rng, 8, 256))
    if kind == "backproject":
        return dict(kind=kind, L=_log_int(rng, 24, 128), B=_log_int(rng, 16, 1024))
    if kind == "mean_add":
        return dict(kind=kind, L=_log_int(rng, 24, 128), B=_log_int(rng, 16, 1024))
    if kind == "cg":
        L = rng.choice([32, 64, 64, 128, rng.randint(24, 100)])
        pre = rng.choice(["none", "diagonal", "circulant"])
        few, most = {"none": (12, 32), "diagonal": (4, 6), "circulant": (8, 12)}[pre]
        return dict(kind=kind, L=L, precond=pre, iters=rng.randint(few, most))
    batch = _log_int(rng, 64, 1024)
    return dict(kind="latent", L=_log_int(rng, 24, 128), r=rng.randint(1, 12), B=rng.randint(64, 1500), batch=batch)


# ----------------------------------------------------------------------------- inputs


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _randn(g, *shape):
    return torch.randn(shape, generator=g, device=DEV)


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device=DEV)


def _axis(m):
    return (torch.arange(m, device=DEV) - m // 2).to(torch.float32)


def _volumes(g, count, L):
    """(count, L^3) smooth random shapes in a ball, with a little white noise, of unit norm."""
    ax = _axis(L)
    r2 = ax[:, None, None] ** 2 + ax[None, :, None] ** 2 + ax[None, None, :] ** 2
    low = torch.exp(-r2 / (2 * (0.12 * L) ** 2))
    ball = torch.sigmoid((0.4 * L - r2.sqrt()))
    out = torch.empty((count, L, L, L), device=DEV)
    for c in range(count):
        v = _randn(g, L, L, L)
        f = torch.fft.fftn(v) * torch.fft.ifftshift(low)
        s = torch.fft.ifftn(f).real
        v = (s / s.std() + 0.05 * v) * ball
        out[c] = v / v.norm()
    return out


def _rotations(g, B):
    q = torch.randn((B, 4), generator=g, device=DEV, dtype=torch.float64)
    w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
    R = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                     2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                     2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], dim=1)
    return R.reshape(B, 3, 3).to(torch.float32)


def _points32(R, L):
    """(B, 3, L^2) float32 frequencies of the central slices, as the reference's pts_rot."""
    k = torch.ceil(torch.arange(L, device=DEV, dtype=torch.float32) - L / 2) / (L / 2) * math.pi
    y, x = (t.reshape(-1) for t in torch.meshgrid(k, k, indexing="ij"))
    p = torch.stack([R[:, d, 0, None] * x + R[:, d, 1, None] * y for d in (2, 1, 0)], dim=1)
    return (torch.remainder(p + math.pi, 2 * math.pi) - math.pi).contiguous()


def _ctf_parameters(g, B):
    """(B, 8): pixel 1.5 A, defocus 1..3 um with some astigmatism, 300 kV, Cs 2.7 mm, contrast 0.1."""
    du = 1e4 + 2e4 * _rand(g, B)
    dv = du + 500 * _randn(g, B)
    one = torch.ones((B,), device=DEV)
    return torch.stack([1.5 * one, du, dv, 180 * _rand(g, B), 300 * one, 2.7 * one, 0.1 * one, 0 * one],
                       dim=1).contiguous()


def _ctf64(params, L):
    """(B, L^2) CTFs of the parameters in 64 bits: the weak-phase form cryo-EM packages use."""
    apix, du, dv, ang, kv, cs, w, ps = params.double().unbind(1)
    V = kv * 1e3
    lam = 12.2639 / torch.sqrt(V + 0.97845e-6 * V * V)
    k = torch.arange(L, device=DEV, dtype=torch.float64) - L // 2
    a, b = (t.reshape(1, -1) for t in torch.meshgrid(k, k, indexing="ij"))
    freq2 = (a * a + b * b) / (L * apix[:, None]) ** 2
    th = 2 * (torch.atan2(b, a) - (ang * math.pi / 180)[:, None])
    df = 0.5 * ((du + dv)[:, None] + (du - dv)[:, None] * torch.cos(th))
    gam = 2 * math.pi * (-0.5 * df * lam[:, None] * freq2 + 0.25 * (cs * 1e7 * lam**3)[:, None] * freq2**2)
    gam = gam - (ps * math.pi / 180)[:, None]
    return torch.sqrt(1 - w * w)[:, None] * torch.sin(gam) - w[:, None] * torch.cos(gam)


def _fft2c(x):
    return torch.fft.fftshift(torch.fft.fft2(torch.fft.ifftshift(x, dim=(-2, -1))), dim=(-2, -1))


def _ifft2c(x):
    return torch.fft.fftshift(torch.fft.ifft2(torch.fft.ifftshift(x, dim=(-2, -1))), dim=(-2, -1))


def _fft3c(x):
    d = (-3, -2, -1)
    return torch.fft.fftshift(torch.fft.fftn(torch.fft.ifftshift(x, dim=d), dim=d), dim=d)


def _ifft3c(x):
    d = (-3, -2, -1)
    return torch.fft.fftshift(torch.fft.ifftn(torch.fft.ifftshift(x, dim=d), dim=d), dim=d)


def _pad3(x, n):
    L = x.shape[-1]
    o = n // 2 - L // 2
    out = torch.zeros(x.shape[:-3] + (n, n, n), dtype=x.dtype, device=x.device)
    out[..., o:o + L, o:o + L, o:o + L] = x
    return out


def _crop3(x, L):
    o = x.shape[-1] // 2 - L // 2
    return x[..., o:o + L, o:o + L, o:o + L]


def _radial_reg(n, noise_var):
    """(n^3) Fourier regulariser, noise over a falling power spectrum."""
    ax = _axis(n)
    k2 = ax[:, None, None] ** 2 + ax[None, :, None] ** 2 + ax[None, None, :] ** 2
    return (noise_var * 1e-3 * (1 + k2 / (0.05 * n) ** 2)).contiguous()


def _inputs(case, seed):
    g = _gen(seed)
    L, kind = case["L"], case["kind"]
    if kind == "step":
        r, B = case["r"], case["B"]
        d = dict(vec=_volumes(g, r, L))
        d["logs"] = math.log(3.0 * L) - 0.1 * torch.arange(r, device=DEV) + 0.05 * _randn(g, r)
        d["rot"] = _rotations(g, B)
        d["pts"] = _points32(d["rot"], L) if case["poses"] == "pts" else None
        d["images"] = _fft2c(_randn(g, B, L, L)).reshape(B, -1).contiguous()
        prm = _ctf_parameters(g, B)
        d["params"] = prm if case["ctf"] == "params" else None
        d["ctf"] = _ctf64(prm, L).float().contiguous() if case["ctf"] == "array" else None
        d["noise_var"] = float(L * L)
        d["fr"] = _radial_reg(L * UPSAMPLE, L * L) if case["reg"] else None
        d["reg_scale"] = 1.0 / 16384 if case["reg"] else 0.0
        return d
    if kind == "autograd":
        r, B = case["r"], case["B"]
        amp = 3.0 * L * torch.exp(-0.1 * torch.arange(r, device=DEV))
        vols = _fft3c(_pad3(_volumes(g, r, L) * amp.reshape(-1, 1, 1, 1), L * UPSAMPLE)).contiguous()
        return dict(vols=vols, pts=_points32(_rotations(g, B), L), images=_fft2c(_randn(g, B, L, L)).contiguous(),
                    ctf=_ctf64(_ctf_parameters(g, B), L).float().reshape(B, L, L), noise_var=float(L * L),
                    fr=_radial_reg(L * UPSAMPLE, L * L), reg_scale=1.0 / 16384)
    if kind == "project":
        r, B = case["r"], case["B"]
        return dict(vols=(_volumes(g, r, L) * 3.0 * L).contiguous(), rot=_rotations(g, B),
                    ctf=_ctf64(_ctf_parameters(g, B), L).float().reshape(B, L, L))
    if kind == "backproject":
        B = case["B"]
        return dict(images=_randn(g, B, L, L), rot=_rotations(g, B),
                    ctf=_ctf64(_ctf_parameters(g, B), L).float().reshape(B, L, L))
    if kind == "mean_add":
        B = case["B"]
        return dict(images=_fft2c(_randn(g, B, L, L)).contiguous(), rot=_rotations(g, B),
                    ctf=_ctf64(_ctf_parameters(g, B), L).float().reshape(B, L, L), offsets=3.0 * _randn(g, B, 2),
                    contrasts=1.0 + 0.1 * _randn(g, B))
    if kind == "cg":
        n = L * UPSAMPLE
        ax = _axis(n)
        z, y, x = torch.meshgrid(ax, ax, ax, indexing="ij")
        k = torch.sqrt(x * x + y * y + z * z)
        u = _randn(g, 3)
        u = u / u.norm()
        # density of slices falling as 1/k, denser around a preferred plane, squared CTFs, plus the
        # half-sets' regulariser, which rises with the frequency.  A fixed number of iterations on a
        # kernel of moderate condition, so that rounding does not decide the iterate
        aniso = 0.15 + torch.exp(-4.0 * ((x * u[0] + y * u[1] + z * u[2]) / (k + 1)) ** 2)
        reg = 1e3 * aniso / (1 + k) * (0.55 + 0.45 * torch.cos(k * k * (20.0 / n**2)))
        reg = (reg + 10.0 * (1 + (k / (0.1 * n)) ** 2)).contiguous()
        truth = _volumes(g, 1, L)[0] * 100
        rhs = reg * _fft3c(_pad3(truth, n)) + torch.sqrt(reg) * _fft3c(_randn(g, n, n, n)) * 0.01
        b = _crop3(_ifft3c(rhs), L).to(torch.complex64).contiguous()
        x0 = _crop3(_ifft3c(rhs / reg), L).real
        return dict(reg=reg, b=b, x0=torch.complex(x0, torch.zeros_like(x0)).contiguous())
    r, B = case["r"], case["B"]
    return dict(vols=_volumes(g, r, L), lam=(9.0 * L * L * torch.exp(-0.2 * torch.arange(r, device=DEV))),
                images=_randn(g, B, L, L), rot=_rotations(g, B),
                ctf=_ctf64(_ctf_parameters(g, B), L).float().reshape(B, L, L), noise_var=1.0)


# ----------------------------------------------------------------------------- the calls


def prepare(case, seed):
    d = _inputs(case, seed)
    L, kind = case["L"], case["kind"]
    s = dict(case=case, d=d)
    if kind == "step":
        # one step object for the whole training, as CovarTrainer.setup_training makes it
        kw = dict(width=case["width"]) if case["disc"] == "nufft" else {}
        s["step"] = cov3d.FusedCovarStep(L, case["r"], case["disc"], UPSAMPLE, device=DEV, max_batch=case["B"],
                                         ls_regulariser=case["objective"] == "ls" and case["reg"], **kw)
        s["gv"], s["gl"] = torch.empty_like(d["vec"]), torch.empty_like(d["logs"])
    elif kind == "autograd":
        s["plan"] = cov3d.NufftPlanDiscretized((L,) * 3, upsample_factor=UPSAMPLE, mode="bilinear")
    elif kind == "project":
        s["plan"] = cov3d.NufftPlan((L,) * 3, batch_size=case["r"], device=DEV)
    elif kind == "backproject":
        s["plan"] = cov3d.NufftPlan((L,) * 3, batch_size=1, device=DEV)
    elif kind == "mean_add":
        s["acc"] = cov3d.MeanBackprojector(L, UPSAMPLE, DEV)
    elif kind == "latent":
        s["data"] = cov3d.ResidentDataset(d["images"], d["rot"], d["ctf"], d["noise_var"])
    return s


def run(s):
    case, d = s["case"], s["d"]
    L, kind = case["L"], case["kind"]
    if kind == "step":  # every batch has its own poses
        step = s["step"]
        if case["poses"] == "rot":
            step.set_rotations(d["rot"])
        else:
            step.set_points(d["pts"])
        c, gv, gl = step(d["vec"], d["logs"], d["images"], d["ctf"], d["noise_var"], d["reg_scale"], d["fr"],
                         0 if case["objective"] == "ml" else 1, grad_vectors=s["gv"], grad_log_sqrt=s["gl"],
                         ctf_params=d["params"])
        return dict(cost=c, grad_vectors=gv, grad_log_sqrt=gl)
    if kind == "autograd":
        s["plan"].setpts(d["pts"])
        vols = d["vols"].detach().requires_grad_()
        c = cov3d.cost_maximum_liklihood_fourier_domain(vols, d["images"], s["plan"], d["ctf"], d["noise_var"],
                                                        d["reg_scale"], d["fr"])
        c.backward()
        return dict(cost=c.detach(), grad=vols.grad)
    if kind == "project":
        s["plan"].setrot(d["rot"])
        return cov3d.vol_forward(d["vols"], s["plan"], d["ctf"])
    if kind == "backproject":
        s["plan"].setrot(d["rot"])
        return cov3d.im_backward(d["images"], s["plan"], d["ctf"])
    if kind == "mean_add":
        s["acc"].grids.zero_()
        s["acc"].add(d["images"], d["ctf"], d["offsets"], d["contrasts"], rotations=d["rot"])
        return s["acc"].grids
    if kind == "cg":
        p = None if case["precond"] == "none" else case["precond"]
        x, info = cov3d.cg_solve(d["reg"], d["b"], d["x0"], L, rtol=1e-12, maxiter=case["iters"], precond=p)
        return dict(x=x, iters=info.iters)
    return cov3d.wiener_coords.latentMAP(s["data"], d["vols"], d["lam"], batch_size=case["batch"])


# ----------------------------------------------------------------------------- work


def _fft3_flops(n, count=1):
    return count * 5.0 * n**3 * 3 * math.log2(n)


def work(case):
    """Each input read once, each output written once; interpolation and spreading at the window's
    cells (4 operations per real weight and complex value), transforms at 5 N log2 N."""
    L, kind = case["L"], case["kind"]
    n, P = L * UPSAMPLE, L * L
    if kind == "cg":
        pre = {"none": 1, "diagonal": 2, "circulant": 1.25}[case["precond"]]
        return dict(bytes=4.0 * n**3 + 24.0 * L**3, flops=case["iters"] * pre * 2 * _fft3_flops(n))
    B, r = case["B"], case.get("r", 1)
    M = B * P
    if kind == "step":
        taps = 8 if case["disc"] == "bilinear" else case["width"] ** 3
        nbytes = 8.0 * r * L**3 + 8.0 * M + (4.0 * M if case["ctf"] == "array" else 32.0 * B)
        nbytes += 36.0 * B if case["poses"] == "rot" else 12.0 * M
        nbytes += 4.0 * n**3 if case["reg"] else 0.0
        flops = 2 * 4.0 * taps * r * M + 2 * _fft3_flops(n, r) + 8.0 * M * (r * (r + 1) / 2 + r + r * r + r)
        return dict(bytes=nbytes, flops=flops)
    if kind == "autograd":
        nbytes = 16.0 * r * n**3 + 4.0 * n**3 + 8.0 * M + 4.0 * M + 12.0 * M
        return dict(bytes=nbytes, flops=2 * 4.0 * 8 * r * M + 8.0 * M * (r * (r + 1) / 2 + r + r * r + r))
    if kind == "project":
        return dict(bytes=4.0 * r * L**3 + 36.0 * B + 4.0 * M + 4.0 * M * r,
                    flops=4.0 * 343 * r * M + _fft3_flops(n, r) + r * B * 10.0 * P * math.log2(L))
    if kind == "backproject":
        return dict(bytes=4.0 * M + 36.0 * B + 4.0 * M + 4.0 * L**3,
                    flops=4.0 * 343 * M + _fft3_flops(n) + B * 10.0 * P * math.log2(L))
    if kind == "mean_add":
        return dict(bytes=8.0 * M + 4.0 * M + 48.0 * B + 2 * 8.0 * n**3, flops=20.0 * M)
    return dict(bytes=4.0 * r * L**3 + 4.0 * M + 4.0 * M + 36.0 * B + 4.0 * B * r,
                flops=4.0 * 343 * r * M + _fft3_flops(n, r) + r * B * 10.0 * P * math.log2(L) + 4.0 * M * r * (r + 3) / 2)


# ----------------------------------------------------------------------------- 64 bits


def _beta(width):
    return 0.97 * math.pi * (1.0 - 1.0 / (2.0 * UPSAMPLE)) * width


def _es(x, width):
    """The exponential-of-semicircle kernel on |x| < width / 2."""
    u = 1.0 - (2.0 * x / width) ** 2
    return torch.where(u > 0, torch.exp(_beta(width) * (torch.sqrt(u.clamp(min=0)) - 1.0)), torch.zeros_like(u))


def _deapodise(L, width):
    """(L) factors per axis: the kernel's Fourier transform (ES), or sinc^2 (bilinear, width 0)."""
    k = (torch.arange(L, device=DEV) - L // 2).double()
    if width == 0:
        return torch.sinc(k / (L * UPSAMPLE)) ** 2
    m = 20000  # midpoint rule of the smooth integrand
    x = (torch.arange(m, device=DEV).double() + 0.5) * (width / 2 / m)
    a = 2 * math.pi * k / (L * UPSAMPLE)
    return 2 * (width / 2 / m) * (torch.cos(a[:, None] * x[None]) * _es(x, width)[None]).sum(1)


def _points64(R, L):
    k = torch.ceil(torch.arange(L, device=DEV, dtype=torch.float64) - L / 2) / (L / 2) * math.pi
    y, x = (t.reshape(-1) for t in torch.meshgrid(k, k, indexing="ij"))
    R = R.double()
    p = torch.stack([R[:, d, 0, None] * x + R[:, d, 1, None] * y for d in (2, 1, 0)], dim=1)
    return torch.remainder(p + math.pi, 2 * math.pi) - math.pi


def _taps(t, n, width):
    """Per axis: cells and weights of the window of fractional index t (M,); width 0: linear with
    zero padding, otherwise ES, periodic."""
    if width == 0:
        c0 = torch.floor(t)
        out = []
        for j, w in ((0, c0 + 1 - t), (1, t - c0)):
            c = c0 + j
            ok = (c >= 0) & (c < n)
            out.append((c.clamp(0, n - 1).long(), torch.where(ok, w, torch.zeros_like(w))))
        return out
    c0 = torch.ceil(t - width / 2)
    return [(torch.remainder(c0 + j, n).long(), _es(t - (c0 + j), width)) for j in range(width)]


def _walk(pts, n, width, visit):
    """visit(point slice, cell index, weight) for every window cell of every point; pts (B, 3, P)."""
    t = (pts.double() * (n / (2 * math.pi)) + n // 2).permute(0, 2, 1).reshape(-1, 3)
    step = 1 << 21
    for lo in range(0, t.shape[0], step):
        sl = slice(lo, min(lo + step, t.shape[0]))
        ax = [_taps(t[sl, d].contiguous(), n, width) for d in range(3)]
        for m0, w0 in ax[0]:
            for m1, w1 in ax[1]:
                m01, w01 = (m0 * n + m1) * n, w0 * w1
                for m2, w2 in ax[2]:
                    visit(sl, m01 + m2, w01 * w2)


def _interp64(grid, pts, n, width):
    """Centered grid (r, n, n, n) at the points: (M, r)."""
    r = grid.shape[0]
    flat = torch.view_as_real(grid.reshape(r, -1).T.contiguous()).reshape(-1, 2 * r)
    out = torch.zeros((pts.shape[0] * pts.shape[2], 2 * r), dtype=torch.float64, device=DEV)

    def visit(sl, idx, w):
        out[sl].addcmul_(flat[idx], w[:, None])

    _walk(pts, n, width, visit)
    return torch.view_as_complex(out.reshape(-1, r, 2))


def _spread64(vals, pts, n, width):
    """The adjoint: (M, r) -> centered grid (r, n, n, n)."""
    r = vals.shape[1]
    v = torch.view_as_real(vals.contiguous()).reshape(-1, 2 * r)
    out = torch.zeros((n**3, 2 * r), dtype=torch.float64, device=DEV)

    def visit(sl, idx, w):
        out.index_add_(0, idx, v[sl] * w[:, None])

    _walk(pts, n, width, visit)
    return torch.view_as_complex(out.reshape(-1, r, 2)).T.reshape(r, n, n, n)


def _epilogue64(B, L, ctf):
    """(M, 1) factor of the projections: CTF, 1 / L, zero Nyquist row and column of even images."""
    f = torch.ones((B, L, L), dtype=torch.float64, device=DEV) if ctf is None else ctf.double().reshape(B, L, L).clone()
    if L % 2 == 0:
        f[:, 0, :] = 0
        f[:, :, 0] = 0
    return f.reshape(-1, 1) / L


def _data_term64(Q, y, s2, objective):
    """Sum over images of the per-image cost of Q (B, P, r), and d cost / d conj(Q)."""
    B, P, r = Q.shape
    gram = torch.empty((B, r, r), dtype=torch.complex128, device=DEV)
    h = torch.empty((B, r), dtype=torch.complex128, device=DEV)
    for lo in range(0, B, 128):
        q = Q[lo:lo + 128]
        gram[lo:lo + 128] = q.mH @ q
        h[lo:lo + 128] = (q.mH @ y[lo:lo + 128, :, None]).squeeze(-1)
    eye = torch.eye(r, dtype=torch.complex128, device=DEV)
    if objective == "ml":
        m, b = gram / s2 + eye, h / s2
        z = torch.linalg.solve(m, b[..., None]).squeeze(-1)
        cost = 0.5 * (-(b.conj() * z).sum(-1).real + torch.linalg.slogdet(m)[1])
        C = (torch.linalg.inv(m).conj() + z.conj()[:, :, None] * z[:, None, :]) / (2 * s2)
        u = -z.conj() / (2 * s2)
    else:
        cost = -2 * h.abs().square().sum(-1) + gram.abs().square().sum((-2, -1))
        cost = cost + 2 * s2 * gram.diagonal(dim1=-2, dim2=-1).real.sum(-1)
        C, u = 2 * gram.conj() + 2 * s2 * eye, -2 * h.conj()
    W = torch.empty_like(Q)
    for lo in range(0, B, 128):
        W[lo:lo + 128] = Q[lo:lo + 128] @ C[lo:lo + 128].transpose(1, 2) + y[lo:lo + 128, :, None] * u[lo:lo + 128, None, :]
    return cost.sum(), W


def _step64(case, d):
    L, r, B, ml = case["L"], case["r"], case["B"], case["objective"] == "ml"
    n, s2, width = L * UPSAMPLE, d["noise_var"], case["width"]
    pts = _points64(d["rot"], L) if case["poses"] == "rot" else d["pts"].double()
    ctf = _ctf64(d["params"], L) if d["ctf"] is None else d["ctf"]
    g1 = _deapodise(L, width)
    gc = g1[:, None, None] * g1[None, :, None] * g1[None, None, :]
    es = torch.exp(d["logs"].double()).reshape(-1, 1, 1, 1)
    V = d["vec"].double() * es
    G = _fft3c(_pad3(V / gc, n))
    f = _epilogue64(B, L, ctf)
    Q = (_interp64(G, pts, n, width) * f).reshape(B, L * L, r)
    total, W = _data_term64(Q, d["images"].to(torch.complex128), s2, case["objective"])
    scale = B if ml else B * float(L) ** 4
    F = _spread64((W / scale).reshape(-1, r) * f, pts, n, width)
    cost = total / scale
    if d["fr"] is not None:
        fr = d["fr"].double()
        if ml:
            coef = d["reg_scale"] / (2 * s2)
            cost = cost + coef * (fr * G.abs().square()).sum()
            F = F + coef * fr * G
        else:
            s = d["reg_scale"] / float(L) ** 4
            X = (G * torch.sqrt(fr)).reshape(n, -1)
            K = X @ X.mH
            cost = cost + s * K.abs().square().sum()
            F = F + 2 * s * (K @ X).reshape(r, n, n, n) * torch.sqrt(fr)
    dV = 2 * _crop3(_ifft3c(F) * float(n) ** 3, L).real / gc
    return dict(cost=cost.reshape(1), grad_vectors=dV * es, grad_log_sqrt=(dV * V).sum((1, 2, 3)))


def _autograd64(case, d):
    L, r, B = case["L"], case["r"], case["B"]
    n, s2 = L * UPSAMPLE, d["noise_var"]
    vols, pts, f = d["vols"].to(torch.complex128), d["pts"].double(), _epilogue64(B, L, d["ctf"])
    Q = (_interp64(vols, pts, n, 0) * f).reshape(B, L * L, r)
    total, W = _data_term64(Q, d["images"].reshape(B, -1).to(torch.complex128), s2, "ml")
    grad = 2 * _spread64((W / B).reshape(-1, r) * f, pts, n, 0)
    fr = d["fr"].double()
    cost = total / B + d["reg_scale"] * (fr * vols.abs().square()).sum() / (2 * s2)
    return dict(cost=cost, grad=grad + d["reg_scale"] * fr * vols / s2)


def _project64(vols, rot, ctf, L, width):
    """(B, r, L, L) real images: the projections' centered inverse transforms."""
    n, B, r = L * UPSAMPLE, rot.shape[0], vols.shape[0]
    g1 = _deapodise(L, width)
    G = _fft3c(_pad3(vols.double() / (g1[:, None, None] * g1[None, :, None] * g1[None, None, :]), n))
    Q = _interp64(G, _points64(rot, L), n, width) * _epilogue64(B, L, ctf)
    return _ifft2c(Q.reshape(B, L * L, r).permute(0, 2, 1).reshape(B, r, L, L)).real


def _backproject64(case, d):
    L, B = case["L"], case["B"]
    n = L * UPSAMPLE
    y = _fft2c(d["images"].double() / L**2).reshape(-1, 1) * _epilogue64(B, L, d["ctf"])
    F = _spread64(y, _points64(d["rot"], L), n, 7)
    g1 = _deapodise(L, 7)
    return _crop3(_ifft3c(F) * float(n) ** 3, L).real / (g1[:, None, None] * g1[None, :, None] * g1[None, None, :])


def _mean_add64(case, d):
    """Nearest cells from the float32 coordinates (the reference's scaling and rounding, which
    decides the cell), sums in 64 bits."""
    L, B = case["L"], case["B"]
    n = L * UPSAMPLE
    w = _points32(d["rot"], L).permute(0, 2, 1).reshape(-1, 3)
    x = w * torch.tensor(n / (n - 1) / math.pi, dtype=torch.float32) + torch.tensor(1 / (n - 1), dtype=torch.float32)
    c = torch.round((x + 1.0) * 0.5 * (n - 1)).long()
    ok = ((c >= 0) & (c < n)).all(1)
    idx = ((c[:, 0] * n + c[:, 1]) * n + c[:, 2])[ok]
    k = torch.ceil(torch.arange(L, device=DEV, dtype=torch.float64) - L / 2) * 2 * math.pi / L
    gy, gx = torch.meshgrid(k, k, indexing="ij")
    o = d["offsets"].double()
    phase = torch.exp(-1j * (gx * o[:, 0].reshape(-1, 1, 1) + gy * o[:, 1].reshape(-1, 1, 1)))
    f = d["ctf"].double() * d["contrasts"].double().reshape(-1, 1, 1)
    nyq = _epilogue64(B, L, None).reshape(-1)
    rhs = (d["images"].to(torch.complex128) * phase * f).reshape(-1) * nyq
    lhs = (f * f / L).reshape(-1) * nyq
    v = torch.stack([rhs.real, rhs.imag, lhs], dim=1)[ok]
    out = torch.zeros((n**3, 3), dtype=torch.float64, device=DEV).index_add_(0, idx, v)
    zero = torch.zeros_like(out[:, 2])
    return torch.stack([torch.complex(out[:, 0], out[:, 1]), torch.complex(out[:, 2], zero)]).reshape(2, n, n, n)


def _circulant64(reg, L):
    """T. Chan's optimal circulant symbol (L, L, L), centered, of the padding operator."""
    n = reg.shape[-1]
    t = torch.fft.ifftn(torch.fft.ifftshift(reg))
    tau = torch.arange(L, device=DEV)
    a, b = (L - tau).double() / L, tau.double() / L
    for ax in range(3):
        shape = [1, 1, 1]
        shape[ax] = L
        t = t.index_select(ax, tau) * a.reshape(shape) + t.index_select(ax, (tau - L) % n) * b.reshape(shape)
    return torch.fft.fftshift(torch.fft.fftn(t).real).clamp(min=1e-30)


def _cg64(case, d):
    L, pre = case["L"], case["precond"]
    n = L * UPSAMPLE
    reg = d["reg"].double()
    sym = _circulant64(reg, L) if pre == "circulant" else None

    def A(v):
        return _crop3(_ifft3c(reg * _fft3c(_pad3(v, n))), L)

    def prec(v):
        if pre == "diagonal":
            return _crop3(_ifft3c(_fft3c(_pad3(v, n)) / reg), L)
        return _ifft3c(_fft3c(v) / sym) if sym is not None else v

    def dot(u, v):
        return torch.vdot(u.reshape(-1), v.reshape(-1))

    x, b = d["x0"].to(torch.complex128), d["b"].to(torch.complex128)
    res = b - A(x)
    z = prec(res)
    p, rz = z.clone(), dot(res, z).real
    for _ in range(case["iters"]):
        ap = A(p)
        alpha = rz / dot(p, ap)
        x = x + alpha * p
        res = res - alpha * ap
        z = prec(res)
        new = dot(res, z).real
        p, rz = z + (new / rz) * p, new
    return dict(x=x.reshape(-1), iters=case["iters"] - 1)


def _latent64(case, d):
    L, r, B = case["L"], case["r"], case["B"]
    linv = torch.diag(1.0 / (d["lam"].double() + 1e-6))
    out = torch.empty((B, r), dtype=torch.float64, device=DEV)
    for lo in range(0, B, 512):
        hi = min(B, lo + 512)
        q = _project64(d["vols"], d["rot"][lo:hi], d["ctf"][lo:hi], L, 7).reshape(hi - lo, r, -1)
        y = d["images"][lo:hi].double().reshape(hi - lo, -1, 1)
        m = q @ q.transpose(1, 2) / d["noise_var"] + linv
        out[lo:hi] = torch.linalg.solve(m, q @ y / d["noise_var"]).squeeze(-1)
    return out


def exact(case, seed):
    d, kind = _inputs(case, seed), case["kind"]
    if kind == "step":
        return _step64(case, d)
    if kind == "autograd":
        return _autograd64(case, d)
    if kind == "project":
        return _project64(d["vols"], d["rot"], d["ctf"], case["L"], 7)
    if kind == "backproject":
        return _backproject64(case, d).unsqueeze(0)
    if kind == "mean_add":
        return _mean_add64(case, d)
    if kind == "cg":
        return _cg64(case, d)
    return _latent64(case, d)
