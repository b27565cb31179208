"""Parity of the CUDA stencils (through the C ABI) with the oracle.

FP64 kernels vs the FP64 oracle: 1e-12 relative (normwise, max |diff| over
max |ref|).  FP32 kernels compute in FP32 and are compared with the FP64
oracle at 2e-5 relative.  Sizes cover the staged (bulk-copy) path, the
direct path (small / odd z lines), ragged grids and the x-chunk wrap.
"""
import numpy as np
import pytest
import torch

import oracle as O
from helpers import TOL_F32, TOL_F64, golden, rel_err
from mgmol_gb300 import capi, synth

pytestmark = pytest.mark.gpu

CASES = [
    ((16, 12, 20), 0.35, 3),   # ragged, direct path for some ops
    ((32, 32, 32), 0.35, 4),   # staged path
    ((24, 16, 40), 0.30, 2),   # ragged staged
    ((8, 8, 8), 0.35, 2),      # tiny: direct path
    ((40, 36, 64), 0.3, 3),    # x chunk not dividing nx
]


def _inputs(n, h, nf, seed=11):
    ll = tuple(n[i] * h for i in range(3))
    psi, _, _ = synth.gaussian_orbitals(n, ll, nf, seed)
    V = synth.gaussian_wells(n, ll, 6, seed)
    return ll, psi, V


def _dev(a, dt):
    return torch.from_numpy(np.ascontiguousarray(a.astype(dt))).cuda()


@pytest.mark.parametrize("n,h,nf", CASES)
@pytest.mark.parametrize("lap", [0, 1, 2, 3, 4])
def test_fd_apply(n, h, nf, lap):
    ll, psi, _ = _inputs(n, h, nf)
    ctx = capi.Context(n, ll)
    ref = O.fd_apply(n, ll, lap, psi)
    out = ctx.fd_apply(_dev(psi, np.float64), lap).cpu().numpy()
    assert rel_err(out, ref) < TOL_F64
    out32 = ctx.fd_apply(_dev(psi, np.float32), lap).cpu().numpy()
    assert rel_err(out32, ref) < TOL_F32


@pytest.mark.parametrize("n,h,nf", CASES)
def test_rhs_mehr(n, h, nf):
    ll, psi, _ = _inputs(n, h, nf)
    ctx = capi.Context(n, ll)
    ref = O.rhs_mehr(n, ll, psi)
    assert rel_err(ctx.rhs_mehr(_dev(psi, np.float64)).cpu().numpy(), ref) < TOL_F64
    assert rel_err(ctx.rhs_mehr(_dev(psi, np.float32)).cpu().numpy(), ref) < TOL_F32


@pytest.mark.parametrize("n,h,nf", CASES)
@pytest.mark.parametrize("lap,apply_B", [(0, 1), (0, 0), (2, 1), (4, 1), (1, 1)])
def test_hpsi(n, h, nf, lap, apply_B):
    ll, psi, V = _inputs(n, h, nf)
    ctx = capi.Context(n, ll)
    ref = O.hpsi(n, ll, lap, psi, V, apply_B=apply_B)
    out = ctx.hpsi(_dev(psi, np.float64), _dev(V, np.float64), lap, bool(apply_B)).cpu().numpy()
    assert rel_err(out, ref) < TOL_F64
    # FP32 orbitals with FP32 and with FP64 potential
    for vdt in (np.float32, np.float64):
        out32 = ctx.hpsi(_dev(psi, np.float32), _dev(V, vdt), lap, bool(apply_B)).cpu().numpy()
        assert rel_err(out32, ref) < TOL_F32


def test_hpsi_matches_reference_golden():
    G = golden()
    n = tuple(int(x) for x in G["stencil_n"])
    ll = tuple(float(x) for x in G["stencil_ll"])
    ctx = capi.Context(n, ll)
    out = ctx.hpsi(_dev(G["stencil_psi"], np.float64), _dev(G["stencil_V"], np.float64)).cpu().numpy()
    assert rel_err(out, G["hpsi_d"]) < TOL_F64
    for t in range(5):
        o = ctx.fd_apply(_dev(G["stencil_psi"], np.float64), t).cpu().numpy()
        assert rel_err(o, G[f"fd{t}_d"]) < TOL_F64


def test_leading_dimension_padding():
    """BlockVector-style padded columns (ld > numpt)."""
    n, h, nf = (32, 16, 24), 0.3, 3
    ll, psi, V = _inputs(n, h, nf)
    np_ = psi.shape[1]
    ld = np_ + 40
    big = torch.zeros((nf, ld), dtype=torch.float64, device="cuda")
    big[:, :np_] = torch.from_numpy(psi).cuda()
    out = torch.full_like(big, 7.0)
    ctx = capi.Context(n, ll)
    ctx.fd_apply(big[:, :np_], 0, out=out[:, :np_])
    ref = O.fd_apply(n, ll, 0, psi)
    assert rel_err(out[:, :np_].cpu().numpy(), ref) < TOL_F64
    assert torch.all(out[:, np_:] == 7.0)


def test_empty_batch_is_a_no_op():
    n = (16, 16, 16)
    ctx = capi.Context(n, (5.6, 5.6, 5.6))
    u = torch.zeros((0, 4096), dtype=torch.float64, device="cuda")
    assert ctx.fd_apply(u, 0).shape == (0, 4096)


# ---------------------------------------------------------------- drop-in ghosted
def _ghosted(u, n, g):
    nf = u.shape[0]
    G = np.zeros((nf, n[0] + 2 * g, n[1] + 2 * g, n[2] + 2 * g), dtype=u.dtype)
    U = u.reshape(nf, *n)
    G[:, g:-g, g:-g, g:-g] = U
    return G


@pytest.mark.parametrize("lap,g", [(0, 1), (1, 1), (2, 2), (3, 3), (4, 4), (0, 2)])
def test_dropin_fdkernel_del2(lap, g):
    n, h, nf = (16, 12, 20), 0.35, 3
    ll, psi, _ = _inputs(n, h, nf)
    Gh = torch.from_numpy(_ghosted(psi, n, g)).cuda()
    capi.trade_boundaries(n, ll, g, Gh, nf)
    B = torch.zeros_like(Gh)
    capi.fdkernel_del2(n, ll, g, lap, Gh, B, nf)
    out = B[:, g:-g, g:-g, g:-g].reshape(nf, -1).cpu().numpy()
    assert rel_err(out, O.fd_apply(n, ll, lap, psi)) < TOL_F64
    # ghosts of the output untouched
    assert float(B[:, :g].abs().max()) == 0.0


def test_dropin_trade_is_periodic_image():
    n, g = (6, 5, 7), 2
    ll = (6 * 0.3, 5 * 0.3, 7 * 0.3)
    rng = np.random.default_rng(3)
    u = rng.standard_normal((2, n[0] * n[1] * n[2]))
    Gh = torch.from_numpy(_ghosted(u, n, g)).cuda()
    capi.trade_boundaries(n, ll, g, Gh, 2)
    ref = np.pad(u.reshape(2, *n), ((0, 0), (g, g), (g, g), (g, g)), mode="wrap")
    assert np.array_equal(Gh.cpu().numpy(), ref)


def test_dropin_rhs_and_transfers():
    n, h, nf = (16, 12, 20), 0.35, 2
    ll, psi, _ = _inputs(n, h, nf)
    g = 1
    Gh = torch.from_numpy(_ghosted(psi, n, g)).cuda()
    capi.trade_boundaries(n, ll, g, Gh, nf)
    R = torch.zeros((nf, n[0] * n[1] * n[2]), dtype=torch.float64, device="cuda")
    capi.fdkernel_rhs_mehr1(n, ll, g, Gh, R, 0, nf)
    assert rel_err(R.cpu().numpy(), O.rhs_mehr(n, ll, psi)) < TOL_F64
    cn = tuple(x // 2 for x in n)
    C = torch.zeros((nf, cn[0] + 2, cn[1] + 2, cn[2] + 2), dtype=torch.float64, device="cuda")
    capi.mgkernel_restrict3d(n, ll, g, Gh, C, nf)
    c_ref = O.restrict(n, ll, psi)
    assert rel_err(C[:, 1:-1, 1:-1, 1:-1].reshape(nf, -1).cpu().numpy(), c_ref) < TOL_F64
    capi.trade_boundaries(cn, ll, g, C, nf)
    F = torch.zeros_like(Gh)
    capi.mgkernel_extend3d(n, ll, g, C, F, nf)
    e_ref = O.extend(n, ll, c_ref)
    assert rel_err(F[:, 1:-1, 1:-1, 1:-1].reshape(nf, -1).cpu().numpy(), e_ref) < TOL_F64


@pytest.mark.parametrize("n", [(9, 10, 12), (10, 11, 16), (17, 33, 128), (70, 37, 64), (12, 20, 1024),
                               (40, 128, 36)])
@pytest.mark.parametrize("lap", [2, 3, 4])
def test_axis_kernel_tiles(n, lap):
    """The FP32 kernel of the radius 2 .. 4 operators at odd row counts, cut
    tiles and x chunks, against the FP64 kernels (H psi, the smoothing sweeps and
    the fused update): FP32 roundings of up to 27 terms, TOL_F32 as above."""
    ll = tuple(0.3 * x for x in n)
    ctx = capi.Context(n, ll)
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    u = torch.randn((3, ctx.npts), generator=g, device="cuda")
    V = torch.randn(ctx.npts, generator=g, device="cuda")
    psi = torch.randn((3, ctx.npts), generator=g, device="cuda")

    def close(a, b):
        return float((a.double() - b).abs().max() / b.abs().max()) < TOL_F32

    assert close(ctx.hpsi(u, V, lap), ctx.hpsi(u.double(), V.double(), lap))
    assert close(ctx.fd_apply(u, lap), ctx.fd_apply(u.double(), lap))
    out = ctx.precond_mg(u, lap, 0, 0.2)
    assert close(out, ctx.precond_mg(u.double(), lap, 0, 0.2))
    a = ctx.precond_update(u, psi.clone(), 0.4, lap, 0, 0.2)
    assert close(a, ctx.precond_update(u.double(), psi.double(), 0.4, lap, 0, 0.2))


@pytest.mark.parametrize("h", [(0.3, 0.3, 0.3), (0.25, 0.3, 0.35), (0.3, 0.25, 0.25)])
@pytest.mark.parametrize("n", [(32, 24, 16), (20, 18, 44)])
def test_spacings(n, h):
    """Equal and unequal spacings along x, y and z."""
    ll = tuple(a * b for a, b in zip(n, h))
    ctx = capi.Context(n, ll)
    rng = np.random.default_rng(3)
    psi, V = rng.standard_normal((2, ctx.npts)), rng.standard_normal(ctx.npts)
    for dt, tol in ((np.float64, TOL_F64), (np.float32, TOL_F32)):
        p, v = psi.astype(dt), V.astype(dt)
        for lap in (0, 1):
            got = ctx.fd_apply(_dev(p, dt), lap).cpu().numpy()
            assert rel_err(got, O.fd_apply(n, ll, lap, p.astype(np.float64))) < tol
            got = ctx.hpsi(_dev(p, dt), _dev(v, dt), lap).cpu().numpy()
            want = O.hpsi(n, ll, lap, p.astype(np.float64), v.astype(np.float64))
            assert rel_err(got, want) < tol
        got = ctx.rhs_mehr(_dev(p, dt)).cpu().numpy()
        assert rel_err(got, O.rhs_mehr(n, ll, p.astype(np.float64))) < tol


@pytest.mark.parametrize("n,nf", [((72, 32, 64), 150), ((37, 20, 64), 330), ((20, 16, 16), 700)])
def test_chunks_of_a_full_launch(n, nf):
    """Blocks that fill the GPU are cut into other x chunks than a few functions:
    the same bits for each function."""
    ctx = capi.Context(n, tuple(0.3 * x for x in n))
    g = torch.Generator(device="cuda").manual_seed(8)
    u = torch.randn((nf, ctx.npts), generator=g, device="cuda")
    V = torch.randn(ctx.npts, generator=g, device="cuda")
    some = torch.tensor([0, nf // 2, nf - 1], device="cuda")
    for dt in (torch.float32, torch.float64):
        a, v = u.to(dt), V.to(dt)
        b = a[some].contiguous()
        assert torch.equal(ctx.hpsi(a, v)[some], ctx.hpsi(b, v))
        for lap in (0, 1):
            assert torch.equal(ctx.fd_apply(a, lap)[some], ctx.fd_apply(b, lap))
            assert torch.equal(ctx.precond_mg(a, lap, 0, 0.2)[some], ctx.precond_mg(b, lap, 0, 0.2))


def _l2(a, ref):
    d = a.astype(np.longdouble) - ref
    return float(np.sqrt((d * d).sum() / (ref * ref).sum()))


def _residual_like(n, h, seed):
    """A Gaussian with 5 % noise and no mean, as residuals of smooth orbitals have."""
    rng = np.random.default_rng(seed)
    x = [np.exp(-0.5 * ((np.arange(m) - m / 2.3) * h / 1.4) ** 2) for m in n]
    u = x[0][:, None, None] * x[1][:, None] * x[2] * (1.0 + 0.05 * rng.standard_normal(n))
    return u - u.mean()


def _sum_axis(u, a, k=1):
    return np.roll(u, -k, a) + np.roll(u, k, a)


def _coefficients(ctx, n, lap, dt, offsets):
    """The operator's coefficients as it has them: what it makes of a unit value."""
    u = np.zeros((1, int(np.prod(n))), dt)
    u[0, 0] = 1.0
    r = ctx.fd_apply(_dev(u, dt), lap).cpu().numpy().reshape(n)
    return [r[o] for o in offsets]


def test_mehrstellen_fp64_error():
    """The FP64 Mehrstellen operator is as close to extended precision as the
    plain order of its sums, (centre, z, y, y-z edges), then the planes beside,
    each product rounded with its sum (4 fields, 5 % for the field)."""
    n, h = (32, 32, 32), 0.25
    ctx = capi.Context(n, tuple(h * x for x in n))
    L = np.longdouble
    c0, fx, fy, fz, yz, xz, xy = _coefficients(ctx, n, 0, np.float64, [
        (0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (0, 1, 1), (1, 0, 1), (1, 1, 0)])

    def neg_lap(u, fma):
        s = [_sum_axis(u, a) for a in range(3)]
        a = fma(yz, _sum_axis(s[1], 2), fma(fy, s[1], fma(fz, s[2], c0 * u)))
        b = fma(xy, s[1], fma(xz, s[2], fx * u))
        return a + np.roll(b, 1, 0) + np.roll(b, -1, 0)

    def fma64(c, x, y):
        return (L(c) * x.astype(L) + y.astype(L)).astype(np.float64)

    err, plain = 0.0, 0.0
    for seed in range(4):
        u = _residual_like(n, h, seed)
        ref = neg_lap(u.astype(L), lambda c, x, y: c * x + y)
        got = ctx.fd_apply(_dev(u.reshape(1, -1), np.float64), 0).cpu().numpy().reshape(n)
        err += _l2(got, ref)
        plain += _l2(neg_lap(u, fma64), ref)
    assert err < 1.05 * plain
