"""Gram / H matrices, FP64 Cholesky, inverse and trace on the GPU vs the
oracle and the restated tests/testGramMatrix.cc checks."""
import numpy as np
import pytest
import torch

import oracle as O
from helpers import TOL_F64, rel_err
from mgmol_gb300 import capi, synth

pytestmark = pytest.mark.gpu


def _dev(a, dt=np.float64):
    return torch.from_numpy(np.ascontiguousarray(a.astype(dt))).cuda()


@pytest.mark.parametrize("n,nf", [((16, 16, 16), 5), ((32, 24, 16), 70), ((16, 16, 16), 130)])
def test_gram_hmat_fp64(n, nf):
    ll = tuple(x * 0.35 for x in n)
    psi, _, _ = synth.gaussian_orbitals(n, ll, nf, 17)
    V = synth.gaussian_wells(n, ll, 8, 17)
    ctx = capi.Context(n, ll)
    S = ctx.gram(_dev(psi)).cpu().numpy()
    S_ref = O.gram(psi, ctx.vel)
    assert rel_err(S, S_ref) < TOL_F64
    assert np.array_equal(S, S.T)
    hp = O.hpsi(n, ll, 0, psi, V)
    H = ctx.hmat(_dev(psi), _dev(hp)).cpu().numpy()
    assert rel_err(H, O.hmat(psi, hp, ctx.vel)) < TOL_F64


def test_gram_fp32_cuda_cores():
    n, nf = (32, 32, 32), 40
    ll = tuple(x * 0.3 for x in n)
    psi, _, _ = synth.gaussian_orbitals(n, ll, nf, 3)
    ctx = capi.Context(n, ll)
    S = ctx.gram(_dev(psi, np.float32), mode=capi.GEMM_FP32).cpu().numpy()
    S_ref = O.gram(psi.astype(np.float32), ctx.vel)
    # FP32 products: 8-term chains, 128-term FP32 sums, double-float total
    assert rel_err(S, S_ref) < 1e-8


def test_cholesky_inverse_trace():
    """testGramMatrix.cc restated: n = 213, L L^T = S to 1e-14, S^-1 S = I."""
    n = 213
    rng = np.random.default_rng(213)
    A = rng.standard_normal((n, n))
    S = A @ A.T / n + np.eye(n)
    ctx = capi.Context((8, 8, 8), (1, 1, 1))
    L = ctx.cholesky(_dev(S)).cpu().numpy()
    assert np.max(np.abs(np.triu(L, 1))) == 0.0
    assert np.max(np.abs(L @ L.T - S)) <= 1e-14 * np.max(np.abs(S)) * n
    info, L_ref = O.potrf(S)
    assert rel_err(L, L_ref) < 1e-12
    Sinv = ctx.inverse_from_cholesky(_dev(L)).cpu().numpy()
    assert np.max(np.abs(Sinv @ S - np.eye(n))) < 1e-12
    H = rng.standard_normal((n, n))
    H = H + H.T
    tr = float(ctx.trace_prod(_dev(H), _dev(Sinv)).cpu()[0])
    ref = O.trace_prod(H, Sinv)
    assert abs(tr - ref) < 1e-12 * max(1.0, abs(ref))


def test_cholesky_reports_not_spd():
    n = 100
    S = np.eye(n)
    S[70, 70] = -2.0
    ctx = capi.Context((8, 8, 8), (1, 1, 1))
    with pytest.raises(capi.MgxError) as e:
        ctx.cholesky(_dev(S))
    assert e.value.status == capi.MGX_NOT_SPD
    assert "71" in str(e.value)
    # the context stays usable
    L = ctx.cholesky(_dev(np.eye(n) * 4.0)).cpu().numpy()
    assert np.allclose(L, 2.0 * np.eye(n))


@pytest.mark.parametrize("n", [64, 130, 512])
def test_gram_pipeline_on_orbitals(n):
    grid = (16, 16, 16)
    ll = (5.6, 5.6, 5.6)
    psi, _, _ = synth.gaussian_orbitals(grid, ll, n, 5, sigma=(0.8, 1.2))
    ctx = capi.Context(grid, ll)
    S = ctx.gram(_dev(psi))
    S_np = S.cpu().numpy()
    w = np.linalg.eigvalsh(S_np)
    if w[0] <= 0:
        pytest.skip("random orbitals not independent at this size")
    L = ctx.cholesky(S)
    Sinv = ctx.inverse_from_cholesky(L).cpu().numpy()
    assert np.max(np.abs(Sinv @ S_np - np.eye(n))) < 1e-9 * np.linalg.cond(S_np)


@pytest.mark.parametrize("n", [64, 213, 512])
def test_theta_from_cholesky(n):
    """theta = S^-1 H by substitution equals the inverse-then-multiply path
    (GramMatrix::computeInverse + ProjectedMatrices::updateTheta) and its
    trace the energy tr(S^-1 H)."""
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n))
    S = A @ A.T / n + np.eye(n)
    H = rng.standard_normal((n, n))
    H = H + H.T
    ctx = capi.Context((8, 8, 8), (1, 1, 1))
    L = ctx.cholesky(_dev(S))
    th, tr = ctx.theta_from_cholesky(L, _dev(H))
    Sinv = O.inverse_from_chol(L.cpu().numpy())
    ref = O.theta(Sinv, H)
    assert rel_err(th.cpu().numpy(), ref) < 1e-12 * max(1.0, np.linalg.cond(S) / 10)
    t = float(tr.cpu()[0])
    tref = O.trace_prod(H, Sinv)
    assert abs(t - tref) < 1e-12 * max(1.0, abs(tref)) * n


@pytest.mark.parametrize("case", ["a", "b"])
def test_gram_hmat_match_reference_golden(case):
    """The GPU's FP64 S and H against the reference's own getLocalOverlap /
    computeLocalProduct and LocalMatrices2DistMatrix (recorded vectors):
    1e-12 relative and the same entries dropped by the 1e-14 filter; for
    FP32 orbitals (split-BF16x3 on the tensor cores) the product tolerance,
    against the reference's USE_MP matrices."""
    from helpers import golden
    g = golden()
    n = tuple(int(x) for x in g[f"sh{case}_n"])
    ll = tuple(float(x) for x in g[f"sh{case}_ll"])
    ctx = capi.Context(n, ll)
    psi = g[f"sh{case}_psi"]
    S = ctx.gram(_dev(psi)).cpu().numpy()
    H = ctx.hmat(_dev(psi), _dev(g[f"sh{case}_hpsi_d"])).cpu().numpy()
    S_ref, H_ref = g[f"sh{case}_S_d"], g[f"sh{case}_H_d"]
    assert rel_err(S, S_ref) < TOL_F64
    assert rel_err(H, H_ref) < TOL_F64
    assert np.array_equal(S == 0, S_ref == 0)
    assert np.array_equal(H == 0, H_ref == 0)
    p32 = _dev(psi, np.float32)
    S32 = ctx.gram(p32, mode=capi.GEMM_BF16X3).cpu().numpy()
    H32 = ctx.hmat(p32, _dev(g[f"sh{case}_hpsi_f"], np.float32), mode=capi.GEMM_BF16X3).cpu().numpy()
    assert rel_err(S32, g[f"sh{case}_S_f"]) < 2e-5
    assert rel_err(H32, g[f"sh{case}_H_f"]) < 2e-5


@pytest.mark.parametrize("n", [2, 64, 130])
def test_cholesky_of_any_exponent(n):
    """Pivots so small that 1 / d overflows; and rows and columns times powers
    of two of 2^-500 to 2^500, which change no bit of the factor but its
    exponents."""
    ctx = capi.Context((8, 8, 8), (1, 1, 1))
    S = np.ldexp(np.eye(n), -1039)
    L = ctx.cholesky(_dev(S)).cpu().numpy()
    assert np.array_equal(L, np.ldexp(np.sqrt(2.0) * np.eye(n), -520))
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n))
    T = A @ A.T / n + np.eye(n)
    k = rng.integers(-500, 501, n)
    L = ctx.cholesky(_dev(T)).cpu().numpy()
    Lk = ctx.cholesky(_dev(np.ldexp(T, k[:, None] + k[None, :]))).cpu().numpy()
    assert np.array_equal(Lk, np.ldexp(L, np.broadcast_to(k[:, None], L.shape)))


def test_pivot_reciprocals():
    """The reciprocal of a pivot d against 1 / d: the second pivot of
    [[d, d], [d, a]] is a - d (d r(d)), so that with a just above d its error
    shows that of r: at most two roundings, of r and of d r, each 2^-53 (and
    half a unit of the square root and of its square here)."""
    ctx = capi.Context((8, 8, 8), (1, 1, 1))
    rng = np.random.default_rng(9)
    for e in (-1000, -500, -3, 0, 1, 7, 500, 1000):
        d = np.ldexp(1.0 + rng.random(32), e)
        d[:4] = np.ldexp([1.0, 2.0 - 2.0 ** -52, 1.0 + 2.0 ** -52, 1.5], e)
        a = d * (1.0 + 2.0 ** -20)
        S = np.zeros((64, 64))
        i = 2 * np.arange(32)
        S[i, i], S[i, i + 1], S[i + 1, i], S[i + 1, i + 1] = d, d, d, a
        p = np.diagonal(ctx.cholesky(_dev(S)).cpu().numpy())[1::2] ** 2
        assert np.all(np.abs(p - (a - d)) <= 2.0 ** -51 * d + 2.0 ** -51 * (a - d)), e


@pytest.mark.parametrize("n", [257, 700, 1000, 2047])
def test_dense_algebra_of_ragged_blocks(n):
    """Several blocks of 256, the last one ragged (down to one row), through the
    slice products, uneven pairs of inverses among them: the factor, the
    inverse, theta and HB against LAPACK's, and a pivot that fails in a late
    block.  S has a condition number of about 5."""
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n))
    S = A @ A.T / n + np.eye(n)
    H = rng.standard_normal((n, n))
    H = H + H.T
    ctx = capi.Context((8, 8, 8), (1, 1, 1))
    L = ctx.cholesky(_dev(S))
    assert rel_err(L.cpu().numpy(), np.linalg.cholesky(S)) < 1e-12
    Sinv = ctx.inverse_from_cholesky(L)
    assert rel_err(Sinv.cpu().numpy(), np.linalg.inv(S)) < 1e-12
    assert torch.equal(Sinv, Sinv.T)
    want = np.linalg.solve(S, H)
    theta, tr = ctx.theta_from_cholesky(L, _dev(H))
    assert rel_err(theta.cpu().numpy(), want) < 1e-12
    assert abs(float(tr) - np.trace(want)) < 1e-12 * n
    assert rel_err(ctx.theta(Sinv, _dev(H)).cpu().numpy(), want) < 1e-12
    HB = S @ H
    assert rel_err(ctx.update_hb(_dev(S), _dev(H)).cpu().numpy(), 0.5 * (HB + HB.T)) < 1e-12
    S[n - 1, n - 1] = -1.0
    with pytest.raises(capi.MgxError) as e:
        ctx.cholesky(_dev(S))
    assert e.value.status == capi.MGX_NOT_SPD and f"minor {n} " in str(e.value)
