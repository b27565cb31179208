"""FP64 products formed from exact bf16 slices on the tensor cores, against
64-bit torch and extended precision: the Gram-type products, Psi Theta and the
residual's column chunks, at the edges of tiles (128 x at most 128, or 64), of the
sums of 192 and 256 values and of the plane chunks, with operands that are not
finite, without memory, and after waits that give up."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _block(nf, npts, seed, spread=8.0):
    """Values whose size varies over 2^-spread .. 1 within a row."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = torch.randn((nf, npts), generator=g, dtype=torch.float64, device="cuda")
    return x * torch.exp2(-spread * torch.rand((nf, npts), generator=g, dtype=torch.float64,
                                               device="cuda"))


def _bound(A, B, K):
    """What |error| of A B^T may be: a slice drops 2^-56 and the products left
    out 6 x 2^-56 of (row maximum x row maximum) per value of K, with random
    signs; FP64 sums (the comparison's too) round at 2^-53.  64 sqrt(K) 2^-53
    covers both with room for the largest of all entries."""
    return 64.0 * K ** 0.5 * 2.0 ** -53 * A.abs().amax(1)[:, None] * B.abs().amax(1)[None, :]


def _product(A, B):
    """A B^T with sums of 256 values of K added up by error-free two-sums, so
    that the comparison's own rounding does not grow with K."""
    hi = torch.zeros((A.shape[0], B.shape[0]), dtype=torch.float64, device="cuda")
    lo = torch.zeros_like(hi)
    for k in range(0, A.shape[1], 256):
        p = A[:, k:k + 256] @ B[:, k:k + 256].T
        t = hi + p
        v = t - hi
        lo += (hi - (t - v)) + (p - v)
        hi = t
    return hi + lo


@pytest.mark.parametrize("nf,n", [(33, (24, 20, 36)), (64, (32, 32, 32)), (95, (16, 20, 18)),
                                  (97, (20, 18, 14)), (129, (14, 16, 18)), (200, (33, 7, 9)),
                                  (64, (112, 108, 104))])
def test_gram_products(nf, n):
    from mgmol_gb300 import capi
    ctx = capi.Context(n, tuple(float(x) for x in n))  # unit volume element
    K = ctx.npts
    psi, hp = _block(nf, K, 1), _block(nf, K, 2)
    S, H = ctx.gram(psi), ctx.hmat(psi, hp)
    for got, a, b in ((S, psi, psi), (H, psi, hp)):
        assert bool(((got - _product(a, b)).abs() <= _bound(a, b, K)).all())
    assert torch.equal(S, S.T)
    # B with work blocks that cut the functions unevenly
    B = ctx.matb(psi, work=torch.empty((min(nf, 50), K), dtype=torch.float64, device="cuda"))
    bp = ctx.rhs_mehr(psi)
    low = (B - _product(psi, bp)).tril().abs() <= _bound(psi, bp, K)
    assert bool(low.all()) and torch.equal(B, B.T)


@pytest.mark.parametrize("nf,n", [(40, (24, 20, 36)), (64, (32, 32, 32)), (97, (20, 18, 14)),
                                  (260, (17, 9, 11)), (520, (8, 10, 12))])
def test_psi_theta(nf, n):
    from mgmol_gb300 import capi
    ctx = capi.Context(n, tuple(float(x) for x in n))
    psi, hp = _block(nf, ctx.npts, 3), _block(nf, ctx.npts, 4)
    theta = _block(nf, nf, 5)
    got = ctx.mult_matrix(psi, theta)
    a, b = psi.T.contiguous(), theta.T.contiguous()
    assert bool(((got.T - a @ b.T).abs() <= _bound(a, b, nf)).all())
    res = ctx.residual(psi, hp, theta, apply_B=False)
    assert bool(((res.T + hp.T - a @ b.T).abs()
                 <= _bound(a, b, nf) + 2.0 ** -51 * (hp.T.abs() + (a @ b.T).abs())).all())
    # a few columns, over the block of H psi
    j0, nc = 5, nf - 9
    out = hp[j0:j0 + nc].clone()
    cols = b[j0:j0 + nc].contiguous()
    ctx.residual_cols(psi, out, cols, apply_B=False, out=out)
    assert torch.equal(out, res[j0:j0 + nc])


def test_scales_and_zeros():
    """Rows of any exponent, subnormal and zero rows among them."""
    from mgmol_gb300 import capi
    n = (32, 32, 20)
    ctx = capi.Context(n, tuple(float(x) for x in n))
    psi = _block(64, ctx.npts, 6)
    e = torch.linspace(-500, 500, 64, device="cuda", dtype=torch.float64).round()
    psi *= torch.exp2(e)[:, None]
    psi[7] = 0.0
    psi[11] = 5e-310  # subnormal
    H = ctx.hmat(psi, psi.flip(0).contiguous())
    ref = psi @ psi.flip(0).T
    ok = (H - ref).abs() <= _bound(psi, psi.flip(0), ctx.npts) + 1e-14
    assert bool(ok.all()) and bool((H[7] == 0).all())


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
def test_not_finite(bad):
    """An operand that is not finite gives what FP64 multiply-adds give."""
    from mgmol_gb300 import capi
    n = (32, 32, 20)
    ctx = capi.Context(n, tuple(float(x) for x in n))
    psi, hp = _block(64, ctx.npts, 7).abs() + 1.0, _block(64, ctx.npts, 8).abs() + 1.0
    hp[5, 77] = bad
    H = ctx.hmat(psi, hp)
    ref = psi @ hp.T
    ref = torch.where(ref.abs() > 1e-14, ref, torch.zeros_like(ref))  # the filter takes NaN to 0
    assert torch.equal(torch.isinf(H), torch.isinf(ref)) and not bool(torch.isnan(H).any())
    assert torch.equal(H[:, 5], ref[:, 5])
    keep = [j for j in range(64) if j != 5]
    assert bool(((H - ref)[:, keep].abs() <= _bound(psi, psi, ctx.npts)[:, keep] * 64).all())
    theta = _block(64, 64, 9).abs() + 1.0
    got = ctx.mult_matrix(hp, theta)
    want = theta.T @ hp
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(torch.isinf(got), torch.isinf(want))


@pytest.mark.parametrize("polls", ["0", "1", "3", "20"])
def test_waits_that_give_up(polls, monkeypatch):
    """With waits of so few polls the pipelines give up at once or on the way:
    the CUDA-core kernels behind them form the products, and the context stays
    usable."""
    from mgmol_gb300 import capi
    n = (32, 32, 20)
    ctx = capi.Context(n, tuple(float(x) for x in n))
    psi, hp = _block(150, ctx.npts, 21), _block(150, ctx.npts, 22)
    theta = _block(150, 150, 23)
    H, out = ctx.hmat(psi, hp), ctx.mult_matrix(psi, theta)
    monkeypatch.setenv("MGX_WAIT_POLLS", polls)
    S2, H2, out2 = ctx.gram(psi), ctx.hmat(psi, hp), ctx.mult_matrix(psi, theta)
    torch.cuda.synchronize()
    monkeypatch.delenv("MGX_WAIT_POLLS")
    assert bool(((S2 - _product(psi, psi)).abs() <= _bound(psi, psi, ctx.npts)).all())
    assert bool(((H2 - H).abs() <= _bound(psi, hp, ctx.npts)).all())
    assert bool(((out2 - out).T.abs() <= _bound(psi.T, theta.T, 150)).all())
    if polls == "0":  # FP64 sums in another order
        assert not torch.equal(H2, H) and not torch.equal(out2, out)
    assert torch.equal(ctx.hmat(psi, hp), H) and torch.equal(ctx.mult_matrix(psi, theta), out)


@pytest.mark.parametrize("polls", ["0", "1", "3", "20"])
def test_waits_that_give_up_in_place(polls, monkeypatch):
    """A product that replaces its target is formed again by the CUDA cores when
    a wait gives up; one that is added to its target cannot be, and then the
    whole target is NaN: nothing finite is wrong."""
    from mgmol_gb300 import capi
    n = (32, 32, 20)
    ctx = capi.Context(n, tuple(float(x) for x in n))
    g = torch.Generator(device="cuda").manual_seed(31)
    A = torch.randn((700, 700), generator=g, dtype=torch.float64, device="cuda")
    S = A @ A.T / 700 + torch.eye(700, dtype=torch.float64, device="cuda")
    L = torch.linalg.cholesky(S)
    H = A + A.T
    psi, hp = _block(150, ctx.npts, 32), _block(150, ctx.npts, 33)
    cols = _block(150, 150, 34)
    want = cols @ psi - hp
    theta_ref = torch.cholesky_solve(H, L)
    # in place: the substitutions, and columns of Psi Theta over the block they leave
    monkeypatch.setenv("MGX_WAIT_POLLS", polls)
    HB, Sinv = ctx.update_hb(S, H), ctx.inverse_from_cholesky(L)
    theta, trace = ctx.theta_from_cholesky(L, H)
    out = hp.clone()
    ctx.residual_cols(psi, out, cols, apply_B=False, out=out)
    torch.cuda.synchronize()
    monkeypatch.delenv("MGX_WAIT_POLLS")
    HB_ref = S @ H
    assert float((HB - 0.5 * (HB_ref + HB_ref.T)).abs().max()) < 1e-11 * float(HB_ref.abs().max())
    assert float((Sinv @ S - torch.eye(700, device="cuda")).abs().max()) < 1e-11
    for got, ref in ((theta, theta_ref), (out, want)):
        nan = torch.isnan(got)
        assert bool((nan | ((got - ref).abs() < 1e-9)).all())
        assert polls != "0" or bool(nan.all())
    assert bool(torch.isnan(trace).any()) == bool(torch.isnan(theta.diagonal()).any())
    assert float((ctx.update_hb(S, H) - HB).abs().max()) < 1e-11 * float(HB.abs().max())


def test_sums_keep_the_low_digits():
    """Rows of one large value, in sums whose items are long: the low digits
    reach the result whole.  Left out are at most six digit products of 2^-56,
    2^-51.4 of x^2 for 1 <= x < 2, and 2^-56 2 of x in each operand; with the
    rounding of the result below 2^-50."""
    from mgmol_gb300 import capi
    n = (64, 64, 64)
    ctx = capi.Context(n, tuple(float(x) for x in n))
    g = torch.Generator(device="cuda").manual_seed(41)
    x = 1.0 + torch.rand(1024, generator=g, dtype=torch.float64, device="cuda")
    psi = torch.zeros((1024, ctx.npts), dtype=torch.float64, device="cuda")
    psi[torch.arange(1024, device="cuda"), 255 * torch.arange(1024, device="cuda")] = x
    S = ctx.gram(psi)
    d = S.diagonal()
    assert float(((d - x * x) / (x * x)).abs().max()) < 2.0 ** -50
    assert int(torch.count_nonzero(S)) == 1024


@pytest.mark.parametrize("peak", [1.0, 1e2, 1e4, 1e6])
def test_error_contract(peak):
    """Rows with one value far above the rest: from slices, an entry is off by
    2^-54 sqrt(K) of the product of the row maxima (six standard deviations
    here); with the slices off, by a few 2^-53 of the sum of the absolute
    products (sums of 32 terms, those of up to 1024 parts added: 64)."""
    from mgmol_gb300 import capi
    n = (32, 32, 32)
    ctx = capi.Context(n, tuple(float(x) for x in n))
    g = torch.Generator(device="cuda").manual_seed(51)
    a = torch.randn((70, ctx.npts), generator=g, dtype=torch.float64, device="cuda")
    b = torch.randn((70, ctx.npts), generator=g, dtype=torch.float64, device="cuda")
    at = torch.randint(0, ctx.npts, (2, 70), generator=g, device="cuda")
    row = torch.arange(70, device="cuda")
    a[row, at[0]], b[row, at[1]] = peak, peak
    ref = _product(a, b)
    norm = a.abs().amax(1)[:, None] * b.abs().amax(1)[None, :]
    tail = 2.0 ** -52 * ref.abs() + 1e-14  # the result's own rounding, the filter
    sliced = (ctx.hmat(a, b) - ref).abs()
    assert bool((sliced <= 6 * 2.0 ** -54 * ctx.npts ** 0.5 * norm + tail).all())
    ctx.set_fp64_slices(False)
    units = (ctx.hmat(a, b) - ref).abs()
    assert bool((units <= 64 * 2.0 ** -53 * (a.abs() @ b.abs().T) + tail).all())
    if peak >= 1e4:  # what the slices cost such rows, and the FP64 units keep
        assert float(units.max()) < 0.1 * float(sliced.max())


def test_psi_theta_keeps_eight_digits():
    """Psi Theta with rows of one dominant value, against extended precision:
    2^-60 sqrt(K) of the product of the maxima (eight standard deviations) and
    the result's rounding; seven digits would be off 2^-52 sqrt(K)."""
    import numpy as np
    from mgmol_gb300 import capi
    n, nf = (17, 9, 11), 260
    ctx = capi.Context(n, tuple(float(x) for x in n))
    g = torch.Generator(device="cuda").manual_seed(52)
    psi = torch.randn((nf, ctx.npts), generator=g, dtype=torch.float64, device="cuda") * 2.0 ** -20
    theta = torch.randn((nf, nf), generator=g, dtype=torch.float64, device="cuda") * 2.0 ** -20
    p, j = torch.arange(ctx.npts, device="cuda"), torch.arange(nf, device="cuda")
    psi[p % nf, p] = 1.0 + psi[p % nf, p]
    theta[(7 * j) % nf, j] = 1.0 + theta[(7 * j) % nf, j]
    got = ctx.mult_matrix(psi, theta).cpu().numpy().astype(np.longdouble)
    a, b = psi.cpu().numpy().astype(np.longdouble), theta.cpu().numpy().astype(np.longdouble)
    rng = np.random.default_rng(52)
    for jj in rng.integers(0, nf, 24):
        pp = rng.integers(0, ctx.npts, 48)
        ref = (b[:, jj][:, None] * a[:, pp]).sum(0)
        size = np.abs(a[:, pp]).max(0) * np.abs(b[:, jj]).max()
        bound = 8 * 2.0 ** -60 * nf ** 0.5 * size + 2.0 ** -52 * np.abs(ref)
        assert np.all(np.abs(got[jj, pp] - ref) <= bound)


def _products(ctx, psi, hp, theta, cols):
    """The Gram-type products (B with a work block that cuts the functions),
    Psi Theta and a residual over its own block, as one list."""
    out = hp[3:3 + cols.shape[0]].clone()
    ctx.residual_cols(psi, out, cols, apply_B=False, out=out)
    work = torch.empty_like(psi)
    return [*ctx.gram_hmat_matb(psi, hp, work=work),
            ctx.matb(psi, work=work[:100]), ctx.mult_matrix(psi, theta), out]


def _chunk_case(seed):
    from mgmol_gb300 import capi
    n, nf = (32, 20, 34), 150  # 170 column tiles of 128 points, the last one whole
    ctx = capi.Context(n, tuple(float(x) for x in n))
    psi, hp = _block(nf, ctx.npts, seed), _block(nf, ctx.npts, seed + 1)
    theta = _block(nf, nf, seed + 2)
    return ctx, psi, hp, theta, theta[:, 5:95].T.contiguous()


@pytest.mark.parametrize("cap", [1, 3 << 20, 20 << 20])
def test_chunks_of_planes(cap, monkeypatch):
    """Planes in chunks of K (sums) and of rows (Psi Theta, the residual), down
    to the smallest ones: the bits of one chunk; and a value that is not finite
    in the last points makes the last chunk alone FP64 sums."""
    ctx, psi, hp, theta, cols = _chunk_case(61)
    want = _products(ctx, psi, hp, theta, cols)
    monkeypatch.setenv("MGX_SLICE_CAP", str(cap))
    for got, w in zip(_products(ctx, psi, hp, theta, cols), want):
        assert torch.equal(got, w)
    psi[17, -1] = float("nan")
    hp2 = hp.clone()
    S, H, B, B2, out, res = _products(ctx, psi, hp2, theta, cols)
    monkeypatch.delenv("MGX_SLICE_CAP")
    first = ctx.npts - 128  # rows of the chunks before the last at the smallest cap
    if cap == 1:
        assert torch.equal(out[:, :first], want[4][:, :first])
        assert torch.equal(res[:, :first], want[5][:, :first])
    assert float((out - want[4])[:, :-1].abs().max()) < 1e-11 * float(want[4].abs().max())
    assert bool(torch.isnan(out[:, -1]).all()) and not bool(torch.isnan(out[:, :-1]).any())
    assert bool(torch.isnan(res[:, -1]).all()) and not bool(torch.isnan(res[:, :-1]).any())
    keep = [i for i in range(150) if i != 17]
    assert float((H - want[1])[keep].abs().max()) < 1e-11 * float(want[1].abs().max())


def test_no_memory_for_the_planes(monkeypatch):
    """Without memory for all planes they come in smaller chunks, and without
    memory for any the CUDA cores form the products; the context goes on."""
    ctx, psi, hp, theta, cols = _chunk_case(71)
    want = _products(ctx, psi, hp, theta, cols)
    del ctx
    ctx, *_ = _chunk_case(71)
    monkeypatch.setenv("MGX_SLICE_ROOM", str(24 << 20))  # the first chunks want more
    for got, w in zip(_products(ctx, psi, hp, theta, cols), want):
        assert torch.equal(got, w)
    monkeypatch.setenv("MGX_SLICE_ROOM", "0")
    for got, w in zip(_products(ctx, psi, hp, theta, cols), want):
        assert not torch.equal(got, w)
        assert float((got - w).abs().max()) < 1e-12 * float(w.abs().max())
    monkeypatch.delenv("MGX_SLICE_ROOM")
    for got, w in zip(_products(ctx, psi, hp, theta, cols), want):
        assert torch.equal(got, w)
