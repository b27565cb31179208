"""The workloads that this framework's speed is judged on, each through the
public calls that a program makes (mgmol_gb300.capi, mgmol_gb300.sweep).

One iteration of MGmol's orbital loop applies H to a block of orbitals, forms
the matrices S, H and B, solves with them, forms the residual, preconditions
it with a V-cycle and moves the orbitals; beside it stand the localized step,
the Poisson solve of the Hartree potential and the training of the learned
preconditioner.  A case is one of these calls, or a whole iteration, on
seeded synthetic orbitals (Gaussians with 5 % noise, Gaussian wells) of the
sizes in this repository's configurations, tests and benchmark.

exact() restates every path in 64-bit torch, without this package.
"""
import math

import numpy as np
import torch

from mgmol_gb300 import capi
from mgmol_gb300.sweep import OrbitalSweep

DEV = "cuda"
DT = {"f64": torch.float64, "f32": torch.float32}
MODES = {"fp64": capi.GEMM_FP64, "fp32": capi.GEMM_FP32, "tf32": capi.GEMM_TF32,
         "bf16x3": capi.GEMM_BF16X3, "fp16x3": capi.GEMM_FP16X3}


def listed():
    return [
        # one small H psi, the size of the tests and of smoke(): a call whose
        # launches count
        dict(name="hpsi_f64_8_on_32", op="hpsi", nx=32, ny=32, nz=32, h=0.35, nfunc=8, dtype="f64",
             lap=0),
        # H psi of the mixed-precision configuration: 8th order, FP32 orbitals
        dict(name="hpsi_f32_8th_512_on_128", op="hpsi", nx=128, ny=128, nz=128, h=0.3, nfunc=512,
             dtype="f32", lap=4),
        # the preconditioned update of the mixed sweep, the benchmark's grid
        dict(name="vcycle_update_f32_64_on_192", op="vcycle", nx=192, ny=192, nz=192, h=0.25,
             nfunc=64, dtype="f32", lap=0, levels=2, update=True, masked=False),
        # S, H and B of the plain FP64 iteration (the energy runs' middle size)
        dict(name="matrices_fp64_256_on_96", op="matrices", nx=96, ny=96, nz=96, h=0.25, nfunc=256,
             mode="fp64"),
        # H psi with S, H and B of the mixed iteration
        dict(name="matrices_bf16x3_512_on_128", op="matrices", nx=128, ny=128, nz=128, h=0.3,
             nfunc=512, mode="bf16x3"),
        # the FP64 algebra of one iteration at the benchmark's number of orbitals
        dict(name="dense_2048", op="dense", nfunc=2048),
        # the residual of the mixed iteration, ragged sizes
        dict(name="residual_bf16x3_257_on_96x80x112", op="residual", nx=96, ny=80, nz=112, h=0.3,
             nfunc=257, mode="bf16x3"),
        # the fused step on localized orbitals, its full configuration
        dict(name="local_1536_on_160", op="local", nx=160, ny=160, nz=160, h=0.3, nfunc=1536,
             rlo=4.0, rhi=8.0),
        # the Hartree potential: one field, many small launches
        dict(name="poisson_f64_96", op="poisson", nx=96, ny=96, nz=96, h=0.25, dtype="f64", lap=0),
        # one training step (loss and gradient) of the learned preconditioner
        dict(name="unet_grad_4_on_64", op="unet", nx=64, ny=64, nz=64, h=0.3, nfunc=4, train=True),
        # whole iterations: plain FP64 and mixed
        dict(name="sweep_plain_64_on_64", op="sweep", nx=64, ny=64, nz=64, h=0.35, nfunc=64,
             kind="plain"),
        dict(name="sweep_mixed_256_on_96", op="sweep", nx=96, ny=96, nz=96, h=0.25, nfunc=256,
             kind="mixed"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, lo, hi, mult):
    """Three dimensions, multiples of mult, of a box that is not too flat."""
    n = _log(rng, lo, hi)
    return [max(mult, mult * round(n * rng.uniform(0.8, 1.25) / mult)) for _ in range(3)]


def _funcs(rng, lo, hi, npts, cap):
    """A number of functions whose block holds at most cap points."""
    return max(1, min(_log(rng, lo, hi), cap // npts))


def draw(rng):
    op = rng.choice(["hpsi", "vcycle", "matrices", "dense", "residual", "local", "poisson", "unet",
                     "sweep"])
    c = dict(op=op)
    if op == "dense":
        c["nfunc"] = _log(rng, 24, 2048)
        return c
    if op == "hpsi":
        n = _dims(rng, 16, 176, rng.choice([1, 2, 4, 16]))
        dt = rng.choice(["f64", "f32"])
        c.update(dtype=dt, lap=rng.choice([0, 0, 1, 2, 4]),
                 nfunc=_funcs(rng, 1, 512, n[0] * n[1] * n[2], 2 ** 27 if dt == "f64" else 2 ** 29))
    elif op == "vcycle":
        lv = rng.choice([1, 2, 2, 3])
        dt = rng.choice(["f64", "f32", "f32"])
        n = _dims(rng, 40, 176, rng.choice([1, 2, 4]) * 2 ** lv)
        c.update(dtype=dt, lap=rng.choice([0, 0, 1, 2, 4]), levels=lv, update=rng.random() < 0.5,
                 masked=rng.random() < 0.3,
                 nfunc=_funcs(rng, 1, 256, n[0] * n[1] * n[2], 2 ** 25 if dt == "f64" else 2 ** 28))
    elif op in ("matrices", "residual"):
        mode = rng.choice(["fp64", "fp64", "bf16x3", "bf16x3", "fp16x3", "tf32", "fp32"])
        n = _dims(rng, 24, 128, rng.choice([1, 2, 4, 8]))
        n[2] = 4 * max(1, round(n[2] / 4)) if mode in ("tf32", "bf16x3", "fp16x3") else n[2]
        npts = n[0] * n[1] * n[2]
        nf = _funcs(rng, 3, 512, npts, 2 ** 28)
        if mode in ("fp64", "fp32"):  # the CUDA-core sizes: N^2 P of 256 orbitals on 96^3 at most
            nf = min(nf, max(2, int(math.sqrt(5.7e10 / npts))))
        c.update(mode=mode, nfunc=nf)
    elif op == "local":
        n = _dims(rng, 72, 160, rng.choice([1, 2, 4]))
        # boxes and their halo have to fit the grid
        rhi = min(8.0, 0.3 * (min(n) - 16) / 2 - 0.6)
        c.update(nfunc=_log(rng, 12, 1536), rlo=round(0.5 * rhi, 3), rhi=round(rhi, 3))
        c["h"] = 0.3
    elif op == "poisson":
        n = _dims(rng, 16, 160, rng.choice([2, 4, 8]))
        c.update(dtype=rng.choice(["f64", "f64", "f32"]), lap=rng.choice([0, 0, 1, 2, 4]))
    elif op == "unet":
        n = _dims(rng, 16, 80, 4)
        c.update(train=rng.random() < 0.6, nfunc=_funcs(rng, 1, 16, n[0] * n[1] * n[2], 2 ** 20))
    else:
        kind = rng.choice(["plain", "mixed"])
        n = _dims(rng, 24, 64 if kind == "plain" else 128, rng.choice([4, 8]))
        cap = 2 ** 24 if kind == "plain" else 2 ** 27
        c.update(kind=kind, h=rng.choice([0.25, 0.3, 0.35]))
        npts = n[0] * n[1] * n[2]
        # at most one orbital in 50 bohr^3: denser blocks of these Gaussians
        # are nearly dependent
        c["nfunc"] = max(4, min(_funcs(rng, 6, 256, npts, cap), int(npts * c["h"] ** 3 / 50)))
    c.update(nx=n[0], ny=n[1], nz=n[2])
    c.setdefault("h", rng.choice([0.25, 0.3, 0.35]))
    return c


# ---------------------------------------------------------------- inputs
def _n(c):
    return (c["nx"], c["ny"], c["nz"])


def _ll(c):
    return tuple(c["h"] * x for x in _n(c))


def _npts(c):
    return c["nx"] * c["ny"] * c["nz"]


def _rng(seed, salt):
    g = torch.Generator(device=DEV)
    g.manual_seed(1000003 * int(seed) + salt)
    return g


def _rand(g, *shape):
    return torch.rand(shape, generator=g, dtype=torch.float64, device=DEV)


def _axis_gauss(n, L, centers, width):
    """exp(-d^2 / (2 width^2)) along one axis, periodic minimum image."""
    x = torch.arange(n, dtype=torch.float64, device=DEV) * (L / n)
    d = x[None, :] - centers[:, None]
    d = d - L * torch.round(d / L)
    return torch.exp(-d * d / (2.0 * width[:, None] ** 2))


def _orbitals(c, seed, dtype):
    """Gaussians of width U[1, 2] bohr at uniform centres, times 1 + 0.05 N(0, 1)."""
    n, ll, nf = _n(c), _ll(c), c["nfunc"]
    g = _rng(seed, 1)
    cen = _rand(g, nf, 3) * torch.tensor(ll, dtype=torch.float64, device=DEV)
    sig = 1.0 + _rand(g, nf)
    ax = [_axis_gauss(n[i], ll[i], cen[:, i], sig).to(dtype) for i in range(3)]
    psi = torch.empty((nf, _npts(c)), dtype=dtype, device=DEV)
    step = max(1, 2 ** 26 // _npts(c))
    for f in range(0, nf, step):
        s = slice(f, min(nf, f + step))
        v = psi[s].view(-1, *n)
        v.normal_(1.0, 0.05, generator=g)
        v.mul_(ax[0][s][:, :, None, None] * ax[1][s][:, None, :, None])
        v.mul_(ax[2][s][:, None, None, :])
    return psi


def _potential(c, seed):
    """16 Gaussian wells of depth U[-2, -0.5] and width 1.5 bohr."""
    n, ll = _n(c), _ll(c)
    g = _rng(seed, 2)
    cen = _rand(g, 16, 3) * torch.tensor(ll, dtype=torch.float64, device=DEV)
    depth = -2.0 + 1.5 * _rand(g, 16)
    w = torch.full((16,), 1.5, dtype=torch.float64, device=DEV)
    ax = [_axis_gauss(n[i], ll[i], cen[:, i], w) for i in range(3)]
    return torch.einsum("k,kx,ky,kz->xyz", depth, *ax).reshape(-1).contiguous()


def _gaussian_overlaps(nf, seed):
    """S, B (positive definite) and H of nf normalized Gaussians, with the
    diagonal that 5 % noise adds."""
    g = _rng(seed, 3)
    cen = _rand(g, nf, 3) * (3.0 * nf ** (1.0 / 3.0))
    sig = 1.0 + _rand(g, nf)
    r2 = (cen[:, None, :] - cen[None, :, :]).square().sum(-1)
    one = torch.eye(nf, dtype=torch.float64, device=DEV)

    def overlap(s):
        t = s[:, None] ** 2 + s[None, :] ** 2
        return (2.0 * s[:, None] * s[None, :] / t) ** 1.5 * torch.exp(-r2 / (2.0 * t))

    S = overlap(sig) + 0.01 * one
    B = overlap(0.98 * sig) * 0.97 + 0.01 * one
    e = -1.0 + 0.8 * _rand(g, nf)
    H = S * (0.5 * (e[:, None] + e[None, :]) + 0.05 * r2.clamp(max=16.0)) + 0.02 * one
    return S.contiguous(), H.contiguous(), B.contiguous()


def _theta(c, seed):
    """A matrix like B^-1 H of a block that has begun to converge: a
    dominant diagonal, and couplings that fall off."""
    nf = c["nfunc"]
    g = _rng(seed, 4)
    t = torch.randn((nf, nf), generator=g, dtype=torch.float64, device=DEV) * (0.1 / math.sqrt(nf))
    return t + torch.diag(-0.3 - 0.7 * _rand(g, nf))


def _regions(c, seed):
    """Centres and radii of localization regions, on the host: centres and the
    order of the radii by the seed, the radii (so the packed size) by the case."""
    r = np.random.default_rng([int(seed), 5])
    cen = r.uniform(0.0, 1.0, (c["nfunc"], 3)) * np.asarray(_ll(c))
    rad = np.random.default_rng(5).uniform(c.get("rlo", 2.5), c.get("rhi", 5.0), c["nfunc"])
    return cen, r.permutation(rad)


def _box(n, h, center, radius):
    """The box of a localization region: its first point and extents."""
    ovr = radius + math.sqrt(3.0 * h * h) + 1e-8
    k = math.ceil(ovr / h) + 2
    ext = [min(2 * k + 1, m) for m in n]
    org = [0 if 2 * k + 1 >= n[i] else (math.floor(center[i] / h) - k) % n[i] for i in range(3)]
    return org, ext


def _packed(c, seed):
    """psi, phi of localized orbitals on their boxes, one after another."""
    n, ll, h = _n(c), _ll(c), c["h"]
    cen, rad = _regions(c, seed)
    g = _rng(seed, 6)
    sig = (1.0 + _rand(g, c["nfunc"])).cpu().numpy()
    lam = (-0.5 + 0.2 * _rand(g, c["nfunc"])).cpu().numpy()
    psi, scale = [], []
    for f in range(c["nfunc"]):
        org, ext = _box(n, h, cen[f], rad[f])
        a = []
        for i in range(3):
            d = (org[i] + np.arange(ext[i])) % n[i] * h - cen[f, i]
            d -= ll[i] * np.round(d / ll[i])
            a.append(np.exp(-d * d / (2.0 * sig[f] ** 2)))
        psi.append(a)
        scale.append(ext[0] * ext[1] * ext[2])
    # one upload of the axes, one outer product per orbital
    flat = torch.from_numpy(np.concatenate([x for a in psi for x in a])).to(DEV)
    out = torch.empty(sum(scale), dtype=torch.float32, device=DEV)
    o = p = 0
    for f, a in enumerate(psi):
        e = [len(x) for x in a]
        x, y, z = flat[p:p + e[0]], flat[p + e[0]:p + e[0] + e[1]], flat[p + e[0] + e[1]:p + sum(e)]
        p += sum(e)
        out[o:o + scale[f]].view(e)[:] = (x[:, None] * y)[:, :, None] * z
        o += scale[f]
    out *= 1.0 + 0.05 * torch.randn(out.shape, generator=g, device=DEV)
    reps = torch.tensor(scale, device=DEV)
    phi = out * torch.repeat_interleave(torch.from_numpy(lam).float().to(DEV), reps)
    return out, phi


def _weights(seed):
    """He-normal weights of the network (FP32)."""
    g = _rng(seed, 7)
    w = [torch.randn(ci * co * 27, generator=g, device=DEV) * math.sqrt(2.0 / (27 * ci))
         for ci, co in _LAYERS]
    return torch.cat(w)


_GAMMA = 0.2


def prepare(c, seed):
    op = c["op"]
    if op == "dense":
        S, H, B = _gaussian_overlaps(c["nfunc"], seed)
        # the dense calls use a context for its workspaces alone
        return dict(c=c, ctx=capi.Context((8, 8, 8), (1.0, 1.0, 1.0)), S=S, H=H, B=B,
                    info=torch.zeros(2, dtype=torch.int32, device=DEV))
    ctx = capi.Context(_n(c), _ll(c))
    st = dict(c=c, ctx=ctx)
    if op == "hpsi":
        psi = _orbitals(c, seed, DT[c["dtype"]])
        st.update(psi=psi, V=_potential(c, seed).to(psi.dtype), out=torch.empty_like(psi))
    elif op == "vcycle":
        dt = DT[c["dtype"]]
        res = _orbitals(c, seed, dt)
        res -= res.mean(dim=1, keepdim=True)
        st.update(res=res, out=_orbitals(c, seed + 500009, dt),
                  scale=0.9 + 0.2 * _rand(_rng(seed, 8), c["nfunc"]), work=torch.empty_like(res))
        if c["masked"]:
            cen, rad = _regions(c, seed)
            st["masks"] = capi.Masks(ctx, c["levels"] + 1, cen, rad, dtype=dt)
    elif op == "matrices":
        dt = torch.float64 if c["mode"] == "fp64" else torch.float32
        st.update(psi=_orbitals(c, seed, dt), V=_potential(c, seed).to(dt))
        st.update(hpsi=torch.empty_like(st["psi"]),
                  work=torch.empty((min(c["nfunc"], 512), ctx.npts), dtype=dt, device=DEV))
    elif op == "residual":
        dt = torch.float64 if c["mode"] == "fp64" else torch.float32
        st.update(psi=_orbitals(c, seed, dt), hpsi=_orbitals(c, seed + 500009, dt),
                  theta=_theta(c, seed))
        st.update(work=torch.empty_like(st["psi"]), out=torch.empty_like(st["psi"]))
    elif op == "local":
        cen, rad = _regions(c, seed)
        m = capi.Masks(ctx, 1, cen, rad, func=0, kind=0, dtype=torch.float32)
        k = capi.Masks(ctx, 1, cen, rad, func=1, kind=1, dtype=torch.float32)
        loc = capi.Local(ctx, m, k)
        psi, phi = _packed(c, seed)
        st.update(loc=loc, psi=psi, phi=phi, V=_potential(c, seed).float(), u=loc.empty(),
                  w=loc.empty())
        # a program tunes the step once for its regions and keeps the choice
        loc.tune(psi, phi, st["V"], 0.05, st["u"], st["w"])
    elif op == "poisson":
        rho = _potential(c, seed)
        st.update(rho=(rho - rho.mean()).to(DT[c["dtype"]]))
        st.update(vh=torch.zeros_like(st["rho"]))
    elif op == "unet":
        net = capi.UNet(ctx)
        net.set_params(_weights(seed))
        x = _orbitals(c, seed, torch.float32)
        x -= x.mean(dim=1, keepdim=True)
        t = _orbitals(c, seed + 500009, torch.float32)
        st.update(net=net, x=x, t=t, out=torch.empty_like(x))
    else:
        mixed = c["kind"] == "mixed"
        dt = torch.float32 if mixed else torch.float64
        sw = OrbitalSweep(ctx, _potential(c, seed), c["nfunc"], mode=c["kind"],
                          gemm=capi.GEMM_BF16X3 if mixed else capi.GEMM_FP64, gamma=_GAMMA)
        st.update(sweep=sw, psi=_orbitals(c, seed, dt))
    return st


def run(st):
    c, ctx = st["c"], st["ctx"]
    op = c["op"]
    if op == "hpsi":
        return ctx.hpsi(st["psi"], st["V"], c["lap"], out=st["out"])
    if op == "vcycle":
        if c["update"]:
            return ctx.precond_update(st["res"], st["out"], 0.5, c["lap"], c["levels"], _GAMMA,
                                      masks=st.get("masks"), work=st["work"],
                                      psi_scale=st["scale"])
        return ctx.precond_mg(st["res"], c["lap"], c["levels"], _GAMMA, masks=st.get("masks"),
                              out=st["out"])
    if op == "matrices":
        mode = MODES[c["mode"]]
        if c["mode"] == "bf16x3":
            S, H, B = ctx.hpsi_gram_hmat_matb(st["psi"], st["V"], st["hpsi"], mode, work=st["work"])
        else:
            ctx.hpsi(st["psi"], st["V"], out=st["hpsi"])
            S, H, B = ctx.gram_hmat_matb(st["psi"], st["hpsi"], mode, work=st["work"])
        return dict(hpsi=st["hpsi"], S=S, H=H, B=B)
    if op == "dense":
        theta, _ = ctx.theta_from_cholesky(ctx.cholesky(st["B"], info=st["info"][0:1]), st["H"])
        L = ctx.cholesky(st["S"], info=st["info"][1:2])
        Sinv = ctx.inverse_from_cholesky(L)
        HB = ctx.update_hb(st["S"], theta)
        return dict(theta=theta, L=L, Sinv=Sinv, HB=HB, energy=ctx.trace_prod(HB, Sinv),
                    info=st["info"])
    if op == "residual":
        return ctx.residual(st["psi"], st["hpsi"], st["theta"], MODES[c["mode"]], work=st["work"],
                            out=st["out"])
    if op == "local":
        return st["loc"].step(st["psi"], st["phi"], st["V"], 0.05, u=st["u"], w=st["w"])
    if op == "poisson":
        st["vh"].zero_()
        r = ctx.mgm(st["vh"], st["rho"], c["lap"], max_sweeps=_POISSON_SWEEPS, tol=_poisson_tol(c))
        return dict(vh=st["vh"], sweeps=r["nb_sweeps"], levels=r["levels"])
    if op == "unet":
        if c["train"]:
            return st["net"].loss_grad(st["x"], st["t"])
        return st["net"].forward(st["x"], out=st["out"])
    e = st["sweep"].run(st["psi"])
    return dict(psi=st["psi"], energy=e)


_POISSON_SWEEPS = 12


def _poisson_tol(c):
    return 1e-8 if c["dtype"] == "f64" else 1e-3


# ---------------------------------------------------------------- work
def _lap_flops(lap):
    return {0: 30, 1: 10, 2: 20, 4: 36}[lap]


def work(c):
    op, nf = c["op"], c.get("nfunc", 1)
    if op == "dense":
        n = float(nf)
        # in: S, H, B; out: theta, L, S^-1, HB.  Two factors, the solves, the
        # inverse (symmetric), S theta
        return dict(bytes=7 * 8 * n * n, flops=n ** 3 * (2 / 3 + 2 + 2 / 3 + 2))
    P = float(_npts(c))
    s = 4 if c.get("dtype") == "f32" or c.get("mode", "fp64") != "fp64" or c.get("kind") == "mixed" \
        or op in ("local", "unet") else 8
    NP = nf * P
    cyc = NP * 1.2 * (4 * (_lap_flops(c.get("lap", 0)) + 4) + 10)
    prod = 2.0 * nf * nf * P
    if op == "hpsi":
        return dict(bytes=2 * NP * s + P * s, flops=NP * (_lap_flops(c["lap"]) + 10))
    if op == "vcycle":
        return dict(bytes=(3 if c["update"] else 2) * NP * s, flops=cyc)
    if op == "matrices":
        return dict(bytes=2 * NP * s + P * s + 24.0 * nf * nf, flops=2 * prod + NP * 50)
    if op == "residual":
        return dict(bytes=3 * NP * s + 8.0 * nf * nf, flops=prod + NP * 10)
    if op == "local":
        r = 0.5 * (c["rlo"] + c["rhi"])
        box = nf * (2 * (r / c["h"] + 4) + 1) ** 3
        return dict(bytes=box * 24 + 4 * P, flops=box * 100)
    if op == "poisson":
        return dict(bytes=2 * P * s, flops=P * 8 / 7 * 6 * 4 * _lap_flops(c["lap"]))
    if op == "unet":
        w = sum(ci * co * 27 / 8.0 ** lv for (ci, co), lv in zip(_LAYERS, _LEVELS))
        return dict(bytes=2 * NP * 4 + 4.0 * 139104, flops=NP * 2 * w * (3 if c["train"] else 1))
    return dict(bytes=2 * NP * s + P * s, flops=3 * prod + cyc + NP * 60 + 5 * float(nf) ** 3)


# ---------------------------------------------------------------- 64-bit restatement
def _h(n, ll):
    return [ll[i] / n[i] for i in range(3)]


def _shift(u, a, k):
    """u at the points k further along axis a (0..2) of (F, nx, ny, nz)."""
    return torch.roll(u, -k, dims=a + 1)


def _axis_sum(u, a, k=1):
    return _shift(u, a, k) + _shift(u, a, -k)


_FD = {1: (1.0, [-1.0]), 2: (1 / 12, [-16.0, 1.0]), 3: (1 / 180, [-270.0, 27.0, -2.0]),
       4: (1 / 5040, [-8064.0, 1008.0, -128.0, 9.0])}


def _mehr_coeffs(h):
    ih = [1.0 / (x * x) for x in h]
    c0 = 16.0 / 12.0 * sum(ih)
    face = [-10.0 / 12.0 * x + 0.125 * c0 for x in ih]
    return c0, face, {(0, 1): -(ih[0] + ih[1]) / 12, (1, 2): -(ih[1] + ih[2]) / 12,
                      (0, 2): -(ih[0] + ih[2]) / 12}


def _neg_lap(u, lap, h):
    if lap == 0:
        c0, face, edge = _mehr_coeffs(h)
        out = c0 * u
        s = [_axis_sum(u, a) for a in range(3)]
        for a in range(3):
            out += face[a] * s[a]
        for (a, b), e in edge.items():
            out += e * _axis_sum(s[a], b)
        return out
    f, w = _FD[lap]
    out = torch.zeros_like(u)
    c0 = 0.0
    for a in range(3):
        for k, x in enumerate(w):
            cf = x * f / (h[a] * h[a])
            out += cf * _axis_sum(u, a, k + 1)
            c0 -= 2.0 * cf
    return out + c0 * u


def _rhs(u):
    return 0.5 * u + (_axis_sum(u, 0) + _axis_sum(u, 1) + _axis_sum(u, 2)) / 12.0


def _jacobi_factor(lap, h):
    s = sum(1.0 / (x * x) for x in h)
    return {0: 1 / (4 / 3 * s), 1: 6 / (2 * s) / 7, 2: 1 / (2.5 * s) / 1.5,
            3: 1 / (49 / 18 * s) / 1.5, 4: 1 / (1435 / 504 * s) / 1.5}[lap]


def _hpsi64(u, V, lap, h):
    return _neg_lap(u, lap, h) + (_rhs(V * u) if lap == 0 else V * u)


def _coarsen(u):
    for a in range(3):
        u = 0.5 * u + 0.25 * _axis_sum(u, a)
        u = u.index_select(a + 1, torch.arange(0, u.shape[a + 1], 2, device=u.device))
    return u


def _refine(u):
    for a in range(3):
        mid = 0.5 * (u + _shift(u, a, 1))
        u = torch.stack((u, mid), dim=a + 2).flatten(a + 1, a + 2)
    return u


def _mask64(n, ll, level, cen, rad, func, dtype):
    """GridMask values of some orbitals at one level, (F, nx, ny, nz)."""
    ax = []
    for i in range(3):
        m = n[i] >> level
        x = np.concatenate(([0.0], np.cumsum(np.full(m - 1, ll[i] / n[i] * (1 << level)))))
        d = x[None, :] - cen[:, i:i + 1]
        d = d - ll[i] * np.round(d / ll[i])
        ax.append(torch.from_numpy(d * d).to(DEV))
    rc = torch.from_numpy(np.asarray(rad)).to(DEV)[:, None, None, None]
    r = (ax[0][:, :, None, None] + ax[1][:, None, :, None] + ax[2][:, None, None, :]).sqrt() / rc
    if func == 0:
        lo = math.exp(-2.0)
        v = torch.where(r > 0.75, (torch.exp(-32.0 * (r - 0.75) ** 2) - lo) / (1.0 - lo),
                        torch.ones_like(r)).float()
    else:
        v = torch.where(r < 0.99999, torch.ones_like(r), (1.0 - r) / (1.0 - 0.99999))
    return torch.where(r <= 1.0, v.to(dtype).double(), torch.zeros_like(r))


def _clamp(u, m):
    return u if m is None else torch.minimum(torch.maximum(u, -m), m)


def _cycle64(f, v, lap, hs, level, levels, masks):
    h, m = hs[level], masks[level]
    jf = _jacobi_factor(lap, h)
    for _ in range(4 if level == levels else 2):
        w = _neg_lap(v, lap, h) - f
        v = _clamp(v - jf * w, m)
    if level == levels:
        return v
    rc = _clamp(_coarsen(_clamp(w, m)), masks[level + 1])
    e = _cycle64(rc, torch.zeros_like(rc), 1, hs, level + 1, levels, masks)
    v = v - _clamp(_refine(e), m)
    for _ in range(2):
        v = _clamp(v - jf * (_neg_lap(v, lap, h) - f), m)
    return v


def _precond64(c, res, seed, lap, levels, masked, dtype):
    n, ll = _n(c), _ll(c)
    hs = [[x * (1 << lv) for x in _h(n, ll)] for lv in range(levels + 1)]
    out = torch.empty(res.shape, dtype=torch.float64, device=DEV)
    cen, rad = _regions(c, seed) if masked else (None, None)
    for s in _slices(c, 8):
        f = res[s].double().view(-1, *n)
        m = [_mask64(n, ll, lv, cen[s], rad[s], 0, dtype) if masked else None
             for lv in range(levels + 1)]
        out[s] = _cycle64(f, _GAMMA * f, lap, hs, 0, levels, m).reshape(f.shape[0], -1)
    return out


def _slices(c, mult=1):
    step = max(1, 2 ** 26 // (_npts(c) * mult))
    return [slice(f, min(c["nfunc"], f + step)) for f in range(0, c["nfunc"], step)]


def _each(c, fn, *blocks):
    """fn on slices of functions as (F, nx, ny, nz) in 64 bits, as one block."""
    out = torch.empty((c["nfunc"], _npts(c)), dtype=torch.float64, device=DEV)
    for s in _slices(c, 4):
        out[s] = fn(*[b[s].double().view(-1, *_n(c)) for b in blocks]).reshape(s.stop - s.start, -1)
    return out


def _product64(A, B, vel):
    """vel A B^T of two blocks, in 64 bits, without a 64-bit copy of either."""
    out = torch.zeros((A.shape[0], B.shape[0]), dtype=torch.float64, device=DEV)
    step = max(4096, 2 ** 27 // A.shape[0])
    for k in range(0, A.shape[1], step):
        out += A[:, k:k + step].double() @ B[:, k:k + step].double().T
    out *= vel
    return torch.where(out.abs() > 1e-14, out, torch.zeros_like(out))


def _matrices64(c, psi, V):
    h = _h(_n(c), _ll(c))
    vel = h[0] * h[1] * h[2]
    V = V.double().view(1, *_n(c))
    hp = _each(c, lambda u: _hpsi64(u, V, 0, h), psi)
    S, H = _product64(psi, psi, vel), _product64(psi, hp, vel)
    return hp, S, H, _product64(psi, _each(c, _rhs, psi), vel)


def _dense64(S, H, B):
    theta = torch.cholesky_solve(H, torch.linalg.cholesky(B))
    L = torch.linalg.cholesky(S)
    Sinv = torch.cholesky_inverse(L)
    HB = S @ theta
    HB = 0.5 * (HB + HB.T)
    return theta, L, Sinv, HB, (HB * Sinv).sum().reshape(1)


def _residual64(c, psi, hpsi, theta):
    out = torch.empty((c["nfunc"], _npts(c)), dtype=torch.float64, device=DEV)
    step = max(4096, 2 ** 27 // c["nfunc"])
    for k in range(0, _npts(c), step):
        out[:, k:k + step] = theta.T @ psi[:, k:k + step].double()
    for s in _slices(c, 4):
        out[s] = _rhs(out[s].view(-1, *_n(c))).reshape(s.stop - s.start, -1) - hpsi[s]
    return out


def _local64(c, seed):
    n, ll, h = _n(c), _ll(c), c["h"]
    psi, phi = _packed(c, seed)
    V = _potential(c, seed).float().double().view(n)
    cen, rad = _regions(c, seed)
    c0, face, edge = _mehr_coeffs(_h(n, ll))
    jf = _jacobi_factor(0, _h(n, ll))
    us, ws = [], []

    def lap(u):  # zero outside the box
        p = torch.nn.functional.pad(u[None], (1, 1) * 3)
        return _neg_lap(p, 0, _h(n, ll))[0, 1:-1, 1:-1, 1:-1]

    def rhs(u):
        p = torch.nn.functional.pad(u[None], (1, 1) * 3)
        return _rhs(p)[0, 1:-1, 1:-1, 1:-1]

    o = 0
    for f in range(c["nfunc"]):
        org, ext = _box(n, h, cen[f], rad[f])
        size = ext[0] * ext[1] * ext[2]
        a, b = psi[o:o + size].double().view(ext), phi[o:o + size].double().view(ext)
        o += size
        ix = [torch.from_numpy((org[i] + np.arange(ext[i])) % n[i]).to(DEV) for i in range(3)]
        v = V[ix[0][:, None, None], ix[1][:, None], ix[2]]
        d2 = []
        for i in range(3):
            x = np.concatenate(([0.0], np.cumsum(np.full(n[i] - 1, ll[i] / n[i]))))
            d = x[(org[i] + np.arange(ext[i])) % n[i]] - cen[f, i]
            d -= ll[i] * np.round(d / ll[i])
            d2.append(torch.from_numpy(d * d).to(DEV))
        r = (d2[0][:, None, None] + d2[1][:, None] + d2[2]).sqrt() / rad[f]
        lo = math.exp(-2.0)
        zero, one = torch.zeros_like(r), torch.ones_like(r)
        m = torch.where(r > 0.75, (torch.exp(-32.0 * (r - 0.75) ** 2) - lo) / (1.0 - lo), one)
        m = torch.where(r <= 1.0, m.float().double(), zero)
        k = torch.where(r < 0.99999, one, (1.0 - r) / (1.0 - 0.99999))
        k = torch.where(r <= 1.0, k.float().double(), zero)
        res = k * (rhs(b - v * a) - lap(a))
        u1 = _clamp(0.05 * res - jf * (lap(0.05 * res) - res), m)
        w = lap(u1) - res
        us.append(_clamp(u1 - jf * w, m).reshape(-1))
        ws.append(_clamp(w, m).reshape(-1))
    return torch.cat(us), torch.cat(ws)


def _poisson_cycle64(f, lap, n, ll, op_ng, ng, depth):
    h = _h(n, ll)
    jf = _jacobi_factor(lap, h)
    v = torch.zeros_like(f)
    for _ in range(2):
        v = v - jf * (_neg_lap(v, lap, h) - f)
    if depth < 10 and all(x % 2 == 0 and x >= 2 * ng for x in n):
        r = _coarsen(_neg_lap(v, lap, h) - f)
        low = {0: 0, 1: 1, 2: 1, 3: 2, 4: 3}[lap]
        e = _poisson_cycle64(r, low, [x // 2 for x in n], ll, max(low, 1), max(op_ng - 1, 1),
                             depth + 1)
        v = v - _refine(e)
    for _ in range(2):
        v = v - jf * (_neg_lap(v, lap, h) - f)
    return v


def _poisson64(c, rho):
    n, ll = _n(c), _ll(c)
    lap = c["lap"]
    h = _h(n, ll)
    rho = rho.double().view(1, *n)
    rhs = _rhs(rho) if lap == 0 else rho
    v = torch.zeros_like(rhs)
    ng = max(lap, 1)
    for _ in range(_POISSON_SWEEPS):
        r = rhs - _neg_lap(v, lap, h)
        if float(r.norm() / rhs.norm()) < _poisson_tol(c):
            break
        v = v + _poisson_cycle64(r, lap, list(n), ll, ng, ng, 0)
    return v.reshape(-1)


_LAYERS = [(1, 16), (16, 32), (32, 64), (64, 32), (32, 16), (16, 1)]
_LEVELS = [0, 1, 2, 2, 1, 0]


def _unet64(c, seed, x, t):
    n = _n(c)
    p = _weights(seed).to(torch.bfloat16).double().requires_grad_(c["train"])
    ws, o = [], 0
    for ci, co in _LAYERS:
        ws.append(p[o:o + ci * co * 27].view(co, ci, 3, 3, 3))
        o += ci * co * 27

    def conv(a, w):  # 27 shifted products: the 64-bit units are slow in any form
        out = 0
        for i in range(27):
            k = (i // 9 - 1, i // 3 % 3 - 1, i % 3 - 1)
            s = torch.roll(a, (-k[0], -k[1], -k[2]), dims=(2, 3, 4))
            out = out + torch.einsum("oc,ncxyz->noxyz", w[:, :, k[0] + 1, k[1] + 1, k[2] + 1], s)
        return out

    def down(a):
        return _coarsen(a.flatten(0, 1)).unflatten(0, a.shape[:2])

    def up(a):
        return _refine(a.flatten(0, 1)).unflatten(0, a.shape[:2])

    x = x.double().view(-1, 1, *n)
    s = x.square().mean(dim=(1, 2, 3, 4), keepdim=True).sqrt()
    a0 = torch.relu(conv(x / s, ws[0]))
    a1 = torch.relu(conv(down(a0), ws[1]))
    a2 = torch.relu(conv(down(a1), ws[2]))
    s1 = torch.relu(up(conv(a2, ws[3])) + a1)
    s0 = torch.relu(up(conv(s1, ws[4])) + a0)
    y = conv(s0, ws[5])
    if not c["train"]:
        return (y * s).reshape(c["nfunc"], -1)
    loss = (y - t.double().view_as(y) / s).square().mean()
    loss.backward()
    return loss.detach().reshape(1), p.grad


def exact(c, seed):
    op = c["op"]
    if op == "dense":
        theta, L, Sinv, HB, e = _dense64(*_gaussian_overlaps(c["nfunc"], seed))
        return dict(theta=theta, L=L, Sinv=Sinv, HB=HB, energy=e, info=None)
    h = _h(_n(c), _ll(c))
    if op == "hpsi":
        dt = DT[c["dtype"]]
        V = _potential(c, seed).to(dt).double().view(1, *_n(c))
        return _each(c, lambda u: _hpsi64(u, V, c["lap"], h), _orbitals(c, seed, dt))
    if op == "vcycle":
        dt = DT[c["dtype"]]
        res = _orbitals(c, seed, dt)
        res -= res.mean(dim=1, keepdim=True)
        out = _precond64(c, res, seed, c["lap"], c["levels"], c["masked"], dt)
        if c["update"]:
            out.mul_(0.5).add_(_orbitals(c, seed + 500009, dt))
            out.mul_((0.9 + 0.2 * _rand(_rng(seed, 8), c["nfunc"]))[:, None])
        return out
    if op == "matrices":
        dt = torch.float64 if c["mode"] == "fp64" else torch.float32
        hp, S, H, B = _matrices64(c, _orbitals(c, seed, dt), _potential(c, seed).to(dt))
        return dict(hpsi=hp, S=S, H=H, B=B)
    if op == "residual":
        dt = torch.float64 if c["mode"] == "fp64" else torch.float32
        return _residual64(c, _orbitals(c, seed, dt), _orbitals(c, seed + 500009, dt),
                           _theta(c, seed))
    if op == "local":
        return _local64(c, seed)
    if op == "poisson":
        rho = _potential(c, seed)
        return dict(vh=_poisson64(c, (rho - rho.mean()).to(DT[c["dtype"]])), sweeps=None,
                    levels=None)
    if op == "unet":
        x = _orbitals(c, seed, torch.float32)
        x -= x.mean(dim=1, keepdim=True)
        return _unet64(c, seed, x, _orbitals(c, seed + 500009, torch.float32))
    # one whole iteration
    dt = torch.float32 if c["kind"] == "mixed" else torch.float64
    psi = _orbitals(c, seed, dt)
    hp, S, H, B = _matrices64(c, psi, _potential(c, seed).to(dt))
    theta, _, _, _, e = _dense64(S, H, B)
    res = _residual64(c, psi, hp, theta)
    out = _precond64(c, res, seed, 0, 2, False, dt).mul_(0.5).add_(psi)
    return dict(psi=out.mul_((1.0 / S.diagonal().sqrt())[:, None]), energy=e)
