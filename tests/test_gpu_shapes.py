"""Kernels at the sizes where their tiling can go wrong (edges of tiles,
remainders, the smallest and largest of a range), against the FP64 oracle.

Error bounds are derived per test from the longest chain of roundings of the
type, before any run."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# A sum of weighted terms (weights summing to one) is a chain of at most 128
# roundings per thread, then FP64; the weight itself holds at most 4 roundings.
# 256 eps of the terms' root-mean-square scale bounds both.
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n,d", [(1, 1), (2, 3), (63, 4), (64, 5), (65, 16), (127, 17), (128, 8), (129, 24), (1000, 33),
                                 (4097, 64), (20011, 63), (30001, 2)])
def test_native_moments_shapes(issm, orc, cuda, dtype, n, d):
    rng = np.random.default_rng(1000 * d + n)
    X = (rng.normal(size=(n, d)) * (1.0 + rng.random(d)) + 3.0 * rng.normal(size=d)).astype(dtype)
    lw = (rng.normal(size=n) - 7.0).astype(dtype)
    if n > 2:
        lw[rng.integers(0, n, size=n // 8)] = -np.inf  # samples of zero weight
        lw[0] = -6.0
    tx, tl = torch.tensor(X, device=cuda), torch.tensor(lw, device=cuda)
    shift = rng.normal(size=d)
    mean, cov = issm.ops.weighted_moments(tx, tl, issm.ops.logweight_summary(tl), torch.tensor(shift, device=cuda))
    em, ec, _ = orc.weighted_moments(X.astype(np.float64).reshape(-1), d, lw.astype(np.float64))
    bound = 256 * float(np.finfo(dtype).eps)
    w = np.exp(lw.astype(np.float64) - lw.max())
    w /= w.sum()
    sd = np.sqrt(np.diag(ec).reshape(-1))
    spread = np.sqrt(w @ (X.astype(np.float64) - shift) ** 2) + np.abs(shift)
    assert np.all(np.abs(mean.cpu().numpy() - em) <= bound * spread)
    # the pass centres on the computed mean, rounded: its error enters squared
    scale = np.outer(sd, sd) + bound * np.outer(spread, spread) + np.finfo(np.float64).tiny
    assert np.all(np.abs(cov.cpu().numpy() - ec.reshape(d, d)) <= bound * scale)
    assert np.array_equal(cov.cpu().numpy(), cov.cpu().numpy().T)


def _factor_bank(issm, orc, rng, d, k, dtype, dev, dof=None):
    loc = (rng.normal(size=(k, d)) * 0.8).astype(dtype)
    A = rng.normal(size=(k, d, d))
    fac = np.linalg.cholesky(A @ A.transpose(0, 2, 1) / d + 0.5 * np.eye(d)).astype(dtype)
    make = (lambda m, L: issm.FactorGaussian(m, L)) if dof is None else (lambda m, L: issm.FactorStudentT(dtype(dof), m, L))
    db = issm.pack_proposals([make(m, L) for m, L in zip(loc, fac)], dev)
    dofs = None if db.dofs is None else db.dofs.double().cpu().numpy()
    ob = orc.BankView(d, orc.GAUSSIAN if dof is None else orc.STUDENT_T, orc.SCALE_FACTOR,
                      db.locations.double().cpu().numpy(), db.scales.double().cpu().numpy(),
                      db.lognormalizers.double().cpu().numpy(), dofs,
                      None if db.range_risk is None else db.range_risk.cpu().numpy())
    return db, ob


# Forward substitution of a factor with condition number below 100 (floor 0.5)
# in FP32: d rows of up to d roundings of terms no larger than |L||z|; the
# bound used by the other FP32 kernels, 2e-5 of max(1, |value|), holds with
# room at d = 64. FP64: the same count of 1.1e-16 roundings, 1e-12.
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n,d,k,dof", [
    (1, 1, 1, None), (31, 3, 2, 4.0), (33, 4, 5, None), (129, 5, 3, None), (127, 8, 17, 6.0), (300, 9, 40, None),
    (1000, 12, 7, 3.0), (4097, 16, 64, None), (5000, 17, 9, None), (513, 24, 33, None), (2049, 32, 50, 5.0),
    (700, 33, 13, None), (257, 48, 9, None), (900, 49, 21, None), (2000, 64, 12, 5.0), (130, 63, 2, None)])
def test_simt_density_shapes(issm, orc, cuda, dtype, n, d, k, dof):
    """Full, partial and generating denominators over the thread-group splits,
    the resident and the chunked bank and every padded dimension."""
    rng = np.random.default_rng(97 * d + k)
    db, ob = _factor_bank(issm, orc, rng, d, k, dtype, cuda, dof)
    x = (1.5 * rng.normal(size=(n, d))).astype(dtype)
    slots = rng.integers(0, k, size=n).astype(np.int32)
    tx, ts = torch.tensor(x, device=cuda), torch.tensor(slots, device=cuda)
    coef = np.log(rng.dirichlet(np.ones(k))).astype(dtype)
    groups = (1 + np.arange(k) % 3).astype(np.int32)
    tc, tg = torch.tensor(coef, device=cuda), torch.tensor(groups, device=cuda)
    tol = 1e-12 if dtype == np.float64 else 2e-5
    for kind, okind in ((issm.native.DENOM_FULL, orc.DENOM_FULL), (issm.native.DENOM_GENERATING, orc.DENOM_GENERATING),
                        (issm.native.DENOM_PARTIAL, orc.DENOM_PARTIAL)):
        den = issm.ops.denominator(kind, tc, groups=tg if kind == issm.native.DENOM_PARTIAL else None)
        fail = issm.ops.new_failures(cuda)
        got, gen = issm.ops.mixture_logdensity(db, den, tx, slots=ts, failures=fail, generating=True)
        exp, egen, _ = orc.mixture_logdensity(ob, x.astype(np.float64).reshape(-1), okind, coef.astype(np.float64),
                                              slots=slots, group_of_slot=groups)
        for a, b in ((got, exp), (gen, egen)):
            assert np.all(np.abs(a.double().cpu().numpy() - b) <= tol * np.maximum(1.0, np.abs(b)))
        assert int(fail[0].item()) == 0


@pytest.mark.parametrize("dtype,d,k", [(np.float32, 3, 4), (np.float32, 16, 64), (np.float32, 24, 9),
                                       (np.float32, 7, 130)])
def test_simt_two_samples_per_thread(issm, cuda, dtype, d, k):
    """The size from which threads own two samples: bitwise the numbers of
    the same rows evaluated in a small call (the per-pair arithmetic and the
    component order are the same; below the split size)."""
    n = 152 * 4 * 4 * 128 + 77
    rng = np.random.default_rng(d)
    props = [issm.FactorGaussian((rng.normal(size=d)).astype(dtype),
                                 (np.eye(d) + np.tril(0.2 * rng.normal(size=(d, d)), -1)).astype(dtype)) for _ in range(k)]
    db = issm.pack_proposals(props, cuda)
    x = torch.randn(n, d, device=cuda, dtype=torch.float32, generator=torch.Generator(device=cuda).manual_seed(1))
    den = issm.ops.denominator(issm.native.DENOM_FULL, torch.zeros(k, device=cuda))
    big = issm.ops.mixture_logdensity(db, den, x)
    m = 152 * 4 * 128 + 5  # one sample per thread, components not split
    for lo in (0, n - m):
        small = issm.ops.mixture_logdensity(db, den, x[lo:lo + m].contiguous())
        assert torch.equal(big[lo:lo + m], small)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n,d,k,dof", [(100, 3, 2, None), (1000, 10, 24, 5.0), (333, 33, 40, None), (4096, 4, 5, None)])
def test_simt_round_draws_and_weights(issm, cuda, dtype, n, d, k, dof):
    """A round's samples equal the separate draw's and its weights the
    separate density's, bitwise up to the component split's merge order."""
    from oracle import oracle as orc
    rng = np.random.default_rng(n + d)
    db, _ = _factor_bank(issm, orc, rng, d, k, dtype, cuda, dof)
    tdt = torch.float32 if dtype == np.float32 else torch.float64
    slots = torch.tensor(rng.integers(0, k, size=n).astype(np.int32), device=cuda)
    normals = torch.tensor(rng.normal(size=n * d).astype(dtype), device=cuda)
    rn = torch.tensor(rng.normal(size=n * 8).astype(dtype), device=cuda) if dof else None
    ru = torch.tensor(rng.random(size=n * 8).astype(dtype), device=cuda) if dof else None
    rad = dict(radial_normals=rn, rn_stride=8, radial_uniforms=ru, ru_stride=8) if dof else {}
    coef = torch.full((k,), -float(np.log(k)), dtype=tdt, device=cuda)
    den = issm.ops.denominator(issm.native.DENOM_FULL, coef)
    db.proposal_ids = torch.arange(1, k + 1, device=cuda)
    x, lw, pid = issm.ops.mis_round(db, den, slots, normals, **rad)
    assert torch.equal(x, issm.ops.draw(db, normals, n, slots=slots, **rad))
    assert torch.equal(lw, -issm.ops.mixture_logdensity(db, den, x, slots=slots))
    assert torch.equal(pid, slots.long() + 1)
    one = issm.ops.draw(db, normals, n, fixed_slot=k - 1, **rad)
    same = issm.ops.draw(db, normals, n, slots=torch.full((n,), k - 1, dtype=torch.int32, device=cuda), **rad)
    eps = float(np.finfo(dtype).eps)
    assert torch.allclose(one, same, rtol=4 * eps, atol=64 * eps)


# The selected elements are exact; the interpolation fraction divides a
# difference of cumulative weights (each within n 1e-16 of its sum of at most
# one) by one sample's weight, at least 1e-3 / n here: below 1e-6 for
# n <= 3e4, and values are compared where neighbouring values are O(1) apart.
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("kind", ["smooth", "equal", "integers", "infinite", "offset", "clusters", "huge"])
@pytest.mark.parametrize("n,d", [(2, 1), (1023, 5), (1025, 3), (30_000, 4)])
def test_weighted_quantile_levels(issm, orc, cuda, dtype, kind, n, d):
    rng = np.random.default_rng(n + d)
    x = rng.normal(size=(n, d))
    if kind == "equal":
        x[:] = 2.5
    elif kind == "integers":
        x = np.round(2.0 * x)
    elif kind == "infinite":
        x[rng.random((n, d)) < 0.2] = np.inf
        x[rng.random((n, d)) < 0.2] = -np.inf
    elif kind == "offset":
        x = 1.0e6 + 1.0e-3 * x
    elif kind == "clusters":
        x = np.where(rng.random((n, d)) < 0.5, 1.0e30, -1.0e-30) * (1.0 + 1.0e-7 * x)
    elif kind == "huge":
        x = x * (1.0e300 if dtype == torch.float64 else 1.0e38)
    lw = rng.uniform(-5.0, 0.0, size=n)
    tx = torch.tensor(x, device=cuda).to(dtype)
    tl = torch.tensor(lw, device=cuda).to(dtype)
    probs = [0.0, 0.05, 0.5, 0.95, 1.0]
    got = issm.quantile(issm.WeightedSamples(tx, tl), probs).cpu().numpy()
    w = np.exp(tl.double().cpu().numpy())
    exp = orc.weighted_quantile(tx.double().cpu().numpy().reshape(-1), d, w / w.sum(), probs)
    nan = np.isnan(exp)  # an interpolation between opposite infinities
    assert np.array_equal(np.isnan(got), nan)
    tol = 1e-6 if dtype == torch.float64 else 2e-6
    with np.errstate(invalid="ignore"):
        ok = (got == exp) | (np.abs(got - exp) <= tol * np.maximum(np.abs(exp), np.minimum(1.0, np.abs(x).max())))
    assert np.all(ok | nan), (got[~(ok | nan)], exp[~(ok | nan)])


def test_weighted_quantile_beyond_kept_weights(issm, cuda):
    """More samples than the workspace keeps weights for: equal to the quantile
    of the same samples' sorted cumulative weights."""
    n = (1 << 21) + 13
    g = torch.Generator(device=cuda).manual_seed(3)
    x = torch.randn(n, 2, device=cuda, dtype=torch.float64, generator=g)
    lw = torch.rand(n, device=cuda, dtype=torch.float64, generator=g)
    got = issm.quantile(issm.WeightedSamples(x, lw), [0.1, 0.5])
    w = torch.softmax(lw, 0)
    for c in range(2):
        v, at = torch.sort(x[:, c])
        cum = torch.cumsum(w[at], 0)
        for j, p in enumerate((0.1, 0.5)):
            thr = p * (cum[-1] - w[at[0]]) + w[at[0]]
            up = int(torch.searchsorted(cum, thr, right=True))
            # within the neighbouring samples, whose distance bounds any interpolation fraction's rounding
            assert float(v[up - 2]) <= float(got[j, c]) <= float(v[up + 1])


@pytest.mark.parametrize("kind", ["logistic", "linreg"])
@pytest.mark.parametrize("form", ["bf16", "tf32", "bf16x1"])
@pytest.mark.parametrize("d,nobs,n", [(2, 1, 127), (16, 255, 128), (17, 256, 129), (32, 1537, 20_000), (33, 31, 40_000),
                                      (64, 512, 39_000), (64, 513, 300), (5, 33, 60_001)])
def test_glm_rows_do_not_depend_on_their_tile(issm, cuda, kind, form, d, nobs, n):
    """Resident and streamed observation tiles, ragged last tiles of both
    kinds, several row tiles per CTA: every row of a call equals, bitwise, the
    same row evaluated in a call of its own few neighbours."""
    rng = np.random.default_rng(nobs + n)
    X = rng.normal(size=(nobs, d))
    beta = rng.normal(size=d) / np.sqrt(d)
    y = (rng.random(nobs) < 0.4).astype(np.float64) if kind == "logistic" else X @ beta + rng.normal(size=nobs)
    t = issm.LogisticRegressionTarget(X, y, 10.0) if kind == "logistic" else issm.LinearRegressionTarget(X, y, 0.5, 2.0)
    prec = {"bf16": issm.native.PREC_BF16, "tf32": issm.native.PREC_TF32, "bf16x1": issm.native.PREC_BF16X1}[form]
    bound = t.bind(cuda, torch.float32)
    x = torch.tensor((beta + 0.3 * rng.normal(size=(n, d))).astype(np.float32), device=cuda)
    got = bound.evaluate(x, precision=prec)
    assert bool(torch.isfinite(got).all())
    for lo in (0, n // 2 - 50, n - 101, n - 1):
        lo = max(lo, 0)
        rows = x[lo:lo + 101].clone()
        assert torch.equal(got[lo:lo + 101], bound.evaluate(rows, precision=prec))
    assert int(issm.native.scoped_workspace(cuda, "glm")[:4].view(torch.int32).item()) == 0


# A linear predictor is a chain of d FP roundings of terms |x_c b_c| and each
# observation adds one more; with u the unit roundoff the log target's error is
# below (d + 8) u sum_o |dl/deta_o| sum_c |x_oc b_c| + 16 u sum_o |l_o|.
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kind", ["logistic", "linreg"])
@pytest.mark.parametrize("d,nobs,n", [(1, 1, 1), (5, 63, 33), (33, 65, 500), (64, 1100, 127), (65, 64, 40), (130, 200, 70),
                                      (12, 50, 10_007), (7, 129, 40_001)])
def test_simt_regression_shapes(issm, cuda, dtype, kind, d, nobs, n):
    rng = np.random.default_rng(d + nobs)
    X = rng.normal(size=(nobs, d)).astype(dtype).astype(np.float64)
    beta = rng.normal(size=d) / np.sqrt(d)
    y = (rng.random(nobs) < 0.4).astype(np.float64) if kind == "logistic" else X @ beta + 0.5 * rng.normal(size=nobs)
    y = y.astype(dtype).astype(np.float64)
    t = issm.LogisticRegressionTarget(X, y, 10.0) if kind == "logistic" else issm.LinearRegressionTarget(X, y, 0.5, 2.0)
    B = (beta + 0.3 * rng.normal(size=(n, d))).astype(dtype)
    tdt = torch.float32 if dtype == np.float32 else torch.float64
    got = t.bind(cuda, tdt).evaluate(torch.tensor(B, device=cuda)).double().cpu().numpy()
    B64, pv = B.astype(np.float64), 10.0 if kind == "logistic" else 2.0
    eta, mag = B64 @ X.T, np.abs(B64) @ np.abs(X.T)
    if kind == "logistic":
        term, slope = y * eta - np.logaddexp(0.0, eta), np.ones_like(eta)
        size = np.abs(y * eta) + np.maximum(eta, 0.0) + 1.0
    else:
        r = y - eta
        term, slope = -0.5 * np.log(2 * np.pi * 0.25) - 2.0 * r * r, 4.0 * np.abs(r) + 1.0
        size = 2.0 * r * r + 1.0
    prior = -0.5 * d * np.log(2 * np.pi * pv) - (B64 ** 2).sum(1) / (2 * pv)
    exp = term.sum(1) + prior
    u = float(np.finfo(dtype).eps) / 2
    bound = (d + 8) * u * (slope * mag).sum(1) + 16 * u * (size.sum(1) + d * (1.0 + (B64 ** 2).sum(1)))
    assert np.all(np.abs(got - exp) <= bound)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("d", [1, 2, 3, 4, 6, 33, 64, 130])
@pytest.mark.parametrize("offset", [0, 1, 2])
def test_gather_rows_and_alignments(issm, cuda, dtype, d, offset):
    n, count = 777, 5003
    src = torch.randn(n * d + offset, device=cuda, dtype=dtype)[offset:].view(n, d)
    anc = torch.randint(1, n + 1, (count,), device=cuda)
    assert torch.equal(issm.ops.gather(src, anc), src[anc - 1])


@pytest.mark.parametrize("n", [1, 4095, 4096, 4097, 70_001])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_resampling_kept_weights(issm, orc, cuda, n, dtype):
    """The fixed-point prefix over whole and ragged scan tiles: bit-exact
    ancestors (the weights formed once and kept)."""
    rng = np.random.default_rng(n)
    lw = (rng.normal(size=n) * 2.0).astype(dtype)
    u = rng.random(size=999)
    tl = torch.tensor(lw, device=cuda)
    got = issm.ops.resample_multinomial(tl, torch.tensor(u, device=cuda)).cpu().numpy()
    assert np.array_equal(got, orc.resample_multinomial_fixed(lw.astype(np.float64), u))
    got = issm.ops.resample_systematic(tl, 0.37, 500).cpu().numpy()
    assert np.array_equal(got, orc.resample_systematic_fixed(lw.astype(np.float64), 0.37, 500))


# The forms' bounds on a log density, as for the other tensor-core densities:
# 5e-5 (BF16 x3) and 4e-3 (TF32) of max(1, |value|).
@pytest.mark.parametrize("form,tol", [("bf16", 5e-5), ("tf32", 4e-3)])
@pytest.mark.parametrize("n,d,k,dof", [(1, 64, 3, None), (127, 33, 5, None), (129, 64, 40, None), (255, 17, 9, 5.0),
                                       (257, 32, 12, None), (513, 16, 17, None), (300, 1, 64, 4.0), (1000, 5, 33, None),
                                       (40_001, 64, 7, None), (79_000, 15, 21, None), (200, 63, 4, 7.0)])
def test_paired_tiles_density(issm, orc, cuda, form, tol, n, d, k, dof):
    """More components than one accumulator holds: odd tile counts, partial
    last chunks, several pairs per CTA, full, prefix and partial denominators."""
    rng = np.random.default_rng(13 * d + k)
    db, ob = _factor_bank(issm, orc, rng, d, k, np.float32, cuda, dof)
    db.attach_inverse_factors()
    x = (1.5 * rng.normal(size=(n, d))).astype(np.float32)
    tx = torch.tensor(x, device=cuda)
    prec = issm.native.PREC_BF16 if form == "bf16" else issm.native.PREC_TF32
    coef = np.log(rng.dirichlet(np.ones(k))).astype(np.float32)
    groups = (1 + np.arange(k) % 2).astype(np.int32)
    tc, tg = torch.tensor(coef, device=cuda), torch.tensor(groups, device=cuda)
    fixed = int(rng.integers(0, k))
    for kind, okind in ((issm.native.DENOM_FULL, orc.DENOM_FULL), (issm.native.DENOM_PARTIAL, orc.DENOM_PARTIAL),
                        (issm.native.DENOM_PREFIX, orc.DENOM_PREFIX)):
        terms = k if kind == issm.native.DENOM_PREFIX else 0
        den = issm.ops.denominator(kind, tc, terms=terms, groups=tg if kind == issm.native.DENOM_PARTIAL else None)
        fail = issm.ops.new_failures(cuda)
        got, gen = issm.ops.mixture_logdensity(db, den, tx, fixed_slot=fixed, failures=fail, generating=True,
                                               precision=prec)
        exp, egen, _ = orc.mixture_logdensity(ob, x.astype(np.float64).reshape(-1), okind, coef.astype(np.float64),
                                              terms=terms, fixed_slot=fixed, group_of_slot=groups)
        for a, b in ((got, exp), (gen, egen)):
            assert np.all(np.abs(a.double().cpu().numpy() - b) <= tol * np.maximum(1.0, np.abs(b)))
        assert int(fail[0].item()) == 0
    issm.ops.check_tensor_core_errors(cuda)


# Cholesky backward error, componentwise: |L L^T - A| <= (d + 2) u sqrt(a_ii a_jj),
# u = eps / 2; l = u_ij / d_j here holds three roundings and the scale sqrt(d) two
# more: 4 (d + 4) eps. The FP32 inverse is built from products of three levels:
# |W L - I| <= 4 d eps |W| |L| |W| |L| componentwise.
@pytest.mark.parametrize("d", [1, 2, 7, 8, 9, 15, 17, 24, 31, 32, 33, 40, 41, 48, 49, 56, 57, 63, 64])
def test_fit_factor_panels(issm, cuda, d):
    rng = np.random.default_rng(50 + d)
    B = rng.normal(size=(d, d)) * 10.0 ** rng.uniform(-3, 3, size=(d, 1))
    cov = B @ B.T + np.diag(rng.uniform(0.1, 1.0, size=d) * np.diag(B @ B.T))
    cov = 0.5 * (cov + cov.T)
    mean, prev = rng.normal(size=d), np.eye(d)
    scale = np.sqrt(np.outer(np.diag(cov), np.diag(cov)))
    dp = 16 if d <= 16 else 32 if d <= 32 else 64
    for dtype, eps in ((torch.float64, 2.0**-52), (torch.float32, 2.0**-23)):
        loc = torch.empty(d, dtype=dtype, device=cuda)
        fac = torch.empty(d, d, dtype=dtype, device=cuda)
        ln = torch.empty(1, dtype=dtype, device=cuda)
        inv = torch.full((dp, dp), float("nan"), dtype=torch.float32, device=cuda)
        fail = issm.ops.new_failures(cuda)
        issm.ops.fit_factor(torch.tensor(mean, device=cuda), torch.tensor(cov, device=cuda),
                            torch.tensor(prev, device=cuda, dtype=dtype), loc, fac, ln, failures=fail,
                            regularization=0.0, out_inverse=inv)
        torch.cuda.synchronize()
        assert int(fail[0].item()) == 0
        L = fac.double().cpu().numpy().T
        assert np.all(np.triu(L, 1) == 0)
        assert np.all(np.abs(L @ L.T - cov) <= 4 * (d + 4) * eps * scale)
        W = inv.double().cpu().numpy()
        assert np.all(W[d:, :] == 0) and np.all(W[:, d:] == 0) and np.all(np.triu(W, 1) == 0)
        W = W[:d, :d]
        G = np.abs(W) @ np.abs(L)
        assert np.all(np.abs(W @ L - np.eye(d)) <= 4 * d * 2.0**-23 * (G @ G))


# The FP64 component density in one dimension, L = 1, mu = 0: the ratio x^2 / nu
# holds at most two roundings (2 eps of it, log1p's condition is below 1), log1p 1.5
# ulp, the final product and sum one each: 5 eps of |c| + (nu + 1) / 2 log1p covers it.
@pytest.mark.parametrize("dof", [1.0, 3.0, 1e6])
def test_f64_student_radius_range(issm, cuda, dof):
    """Ratios from 0 and the subnormals through every table interval and its edges
    to the largest finite ones."""
    rng = np.random.default_rng(3)
    j = np.arange(-4, 260)
    edges = np.concatenate([np.ldexp(1.0 + np.clip(j, 0, 255) / 128.0, e) - 1.0 for e in (0, 1, 7, 52, 53, 60)])
    edges = np.concatenate([np.nextafter(edges, 0), edges, np.nextafter(edges, np.inf)])
    wide = np.exp(rng.uniform(np.log(1e-290), np.log(1e290), size=4096))
    ratio = np.concatenate([[0.0, 2.0**-53, 2.0**-52, 0.5, 1.0], np.abs(edges), wide])
    x = np.sqrt(ratio * dof)
    one = np.ones((1, 1))
    db = issm.pack_proposals([issm.FactorStudentT(np.float64(dof), np.zeros(1), one)], cuda)
    den = issm.ops.denominator(issm.native.DENOM_FULL, torch.zeros(1, device=cuda, dtype=torch.float64))
    got = issm.ops.mixture_logdensity(db, den, torch.tensor(x[:, None], device=cuda)).cpu().numpy()
    c = float(db.lognormalizers[0].item())
    xl = x.astype(np.longdouble)
    radial = (np.longdouble(dof + 1.0) / 2.0 * np.log1p(xl * xl / dof)).astype(np.float64)
    assert np.all(np.abs(got - (c - radial)) <= 5 * 2.0**-52 * (abs(c) + radial))


# A log-sum-exp of K terms: each exponential 0.51 ulp plus its argument's rounding
# (half an ulp of a gap below 37.5: 2^-48 of the term, 64 eps / 4), each sum one rounding;
# (16 + K) eps of the sum and 2 eps of the value.
@pytest.mark.parametrize("k", [2, 5, 40, 130])
def test_f64_log_sum_exp(issm, cuda, k):
    rng = np.random.default_rng(k)
    db = issm.pack_proposals([issm.FactorGaussian(np.zeros(2), np.eye(2)) for _ in range(k)], cuda)
    x = rng.normal(size=(700, 2))
    for coef in (np.zeros(k), -40.0 * rng.random(k), -np.arange(k) * np.log(2.0) / 128.0,
                 np.where(np.arange(k) % 3 == 1, -np.inf, -800.0 * rng.random(k))):
        den = issm.ops.denominator(issm.native.DENOM_FULL, torch.tensor(coef, device=cuda))
        got = issm.ops.mixture_logdensity(db, den, torch.tensor(x, device=cuda)).cpu().numpy()
        xl = x.astype(np.longdouble)
        lq = -np.log(2 * np.longdouble(np.pi)) - 0.5 * (xl * xl).sum(1)
        m = coef.max()
        want = (lq + m + np.log(np.exp((coef - m).astype(np.longdouble)).sum())).astype(np.float64)
        assert np.all(np.abs(got - want) <= 2.0**-52 * (16 + k + 4 * (np.abs(want) + abs(m) + np.abs(lq.astype(np.float64)))))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("size", [1, 3, 500, 4099])
def test_round_summary_checks_new_targets(issm, cuda, dtype, size):
    """Invalid targets recorded by the weights' pass of a native run: the failure
    words, round ids and summaries of the separate check."""
    d = 2
    target = issm.QuadraticTarget(np.zeros(d), float("nan"))
    p = issm.FactorGaussian(np.zeros(d, dtype=dtype), np.eye(d, dtype=dtype))
    out = []
    for body in (issm.sampler._native_body, lambda s: issm.sampler._moment_body(s, False)):
        s = issm.prepare_sampler(3, target, issm.AMIS(p, rounds=3, round_size=size), device=cuda, graphs=False)
        body(s)
        torch.cuda.synchronize()
        out.append((s.round_failures.cpu(), s.round_ids.cpu(), s.summaries[0].cpu()))
    assert int(out[0][0][0, 0]) >= size and int(out[0][1].abs().sum()) == 0
    for a, b in zip(*out):
        assert torch.equal(a.nan_to_num(nan=-1.0) if a.is_floating_point() else a,
                           b.nan_to_num(nan=-1.0) if b.is_floating_point() else b)


@pytest.mark.parametrize("d", [5, 8, 12, 16, 24, 33, 40, 64])
@pytest.mark.parametrize("n", [1, 127, 300, 20001])
def test_row_access_widths(issm, cuda, d, n):
    """Samples on 4- and 16-byte boundaries (read 4 and 16 bytes at a time) give
    bitwise the numbers of the aligned array: density of one and of several
    components, the paired tiles and the moments."""
    rng = np.random.default_rng(d)
    gen = torch.Generator(device=cuda).manual_seed(n)
    x = torch.randn(n, d, device=cuda, generator=gen)
    lw = torch.randn(n, device=cuda, generator=gen)
    shift = torch.tensor(0.1 * rng.normal(size=d), device=cuda)

    def offset(k):
        base = torch.empty(n * d + 8, device=cuda)
        y = base[k:k + n * d].view(n, d)
        y.copy_(x)
        return y

    def numbers(y, prec):
        out = list(issm.ops.weighted_moments(y, lw, issm.ops.logweight_summary(lw), shift, precision=prec))
        for k in (1, 3, 21):
            out.append(issm.ops.mixture_logdensity(banks[k], issm.ops.denominator(
                issm.native.DENOM_FULL, torch.zeros(k, device=cuda)), y, precision=prec))
        return [t.clone() for t in out]

    banks = {}
    for k in (1, 3, 21):
        props = [issm.FactorGaussian(rng.normal(size=d).astype(np.float32),
                                     (np.eye(d) + 0.1 * np.tril(rng.normal(size=(d, d)), -1)).astype(np.float32))
                 for _ in range(k)]
        banks[k] = issm.pack_proposals(props, cuda)
        banks[k].attach_inverse_factors()
    for prec in (issm.native.PREC_BF16, issm.native.PREC_TF32):
        want = numbers(x, prec)
        for off in (1, 4):
            for a, b in zip(want, numbers(offset(off), prec)):
                assert torch.equal(a, b)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n,d,k,terms,dof", [(100, 3, 8, 3, None), (5000, 16, 8, 3, 5.0), (1000, 12, 40, 1, None),
                                             (700, 24, 8, 3, None), (333, 33, 60, 2, 4.0), (200_003, 7, 9, 4, None),
                                             (257, 64, 70, 65, None)])
def test_prefix_round_draws_every_slot(issm, orc, cuda, dtype, n, d, k, terms, dof):
    """A round over a prefix of the bank whose samples come from every slot: the
    draws of slots beyond the prefix equal the separate draw's, the weights the
    separate prefix density's, bitwise, and the oracle's (tolerances as
    test_simt_density_shapes)."""
    rng = np.random.default_rng(n + terms)
    db, ob = _factor_bank(issm, orc, rng, d, k, dtype, cuda, dof)
    tdt = torch.float32 if dtype == np.float32 else torch.float64
    slots = rng.integers(0, k, size=n).astype(np.int32)
    slots[:k] = np.arange(k)
    ts = torch.tensor(slots, device=cuda)
    normals = torch.tensor(rng.normal(size=n * d).astype(dtype), device=cuda)
    rad = {}
    if dof:
        rad = dict(radial_normals=torch.tensor(rng.normal(size=n * 8).astype(dtype), device=cuda), rn_stride=8,
                   radial_uniforms=torch.tensor(rng.random(size=n * 8).astype(dtype), device=cuda), ru_stride=8)
    coef = np.log(rng.dirichlet(np.ones(k))).astype(dtype)
    tc = torch.tensor(coef, device=cuda)
    den = issm.ops.denominator(issm.native.DENOM_PREFIX, tc, terms=terms)
    db.proposal_ids = torch.arange(1, k + 1, device=cuda)
    fail = issm.ops.new_failures(cuda)
    x, lw, pid = issm.ops.mis_round(db, den, ts, normals, failures=fail, **rad)
    assert torch.equal(x, issm.ops.draw(db, normals, n, slots=ts, **rad))
    assert torch.equal(lw, -issm.ops.mixture_logdensity(db, den, x, slots=ts))
    assert torch.equal(pid, ts.long() + 1) and int(fail[0].item()) == 0
    exp, _, _ = orc.mixture_logdensity(ob, x.double().cpu().numpy().reshape(-1), orc.DENOM_PREFIX,
                                       coef.astype(np.float64), terms=terms, slots=slots)
    tol = 1e-12 if dtype == np.float64 else 2e-5
    assert np.all(np.abs(lw.double().cpu().numpy() + exp) <= tol * np.maximum(1.0, np.abs(exp)))


# The cumulative weights are sums of at most n positive FP64 terms of total one, in
# any order: (n + 8) eps covers them, the weights' own roundings and the threshold's.
# Within that much weight of the exact threshold lie the only samples that a
# quantile may be formed from, and an interpolation stays between two neighbours.
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("kind", ["narrow", "tiny_top", "tiny_both", "ties"])
@pytest.mark.parametrize("n", [300, 4000, 30_000])
def test_weighted_quantile_between_neighbours(issm, cuda, dtype, kind, n):
    """Weights that span more than forty in the logarithm, the largest or the
    smallest values next to weightless: every quantile lies between the samples
    that hold its threshold."""
    rng = np.random.default_rng(n)
    probs = [0.0, 1e-12, 0.05, 0.5, 0.95, 1.0 - 1e-12, 1.0]
    eps = 2.0**-52
    for rep in range(4):
        x = 3.0 * rng.normal(size=n)
        if kind == "ties":
            x = np.round(2.0 * x) / 2.0
        lw = -1.5 * x * x
        if kind in ("tiny_top", "tiny_both"):
            small = (x > np.quantile(x, 0.9)) | ((x < np.quantile(x, 0.1)) & (kind == "tiny_both"))
            lw = np.where(small, -45.0 - 10.0 * rng.random(n), rng.normal(size=n))
        d = 24  # affine images: other bins for the same order or its reverse
        X = x[:, None] * rng.uniform(0.3, 3.0, size=d) * rng.choice([-1.0, 1.0], size=d) + 5.0 * rng.normal(size=d)
        tx, tl = torch.tensor(X, device=cuda).to(dtype), torch.tensor(lw, device=cuda).to(dtype)
        got = issm.quantile(issm.WeightedSamples(tx, tl), probs).cpu().numpy()
        l64 = tl.double().cpu().numpy()
        w = np.exp((l64 - l64.max()).astype(np.longdouble))
        w /= w.sum()
        V = tx.double().cpu().numpy()
        delta = (n + 8) * eps
        for c in range(d):
            at = np.argsort(V[:, c], kind="stable")
            v, cum = V[at, c], np.cumsum(w[at])
            for j, p in enumerate(probs):
                thr = np.longdouble(p) * (cum[-1] - w[at[0]]) + w[at[0]]
                lo = max(int(np.searchsorted(cum, thr - delta, side="right")) - 1, 0)
                hi = min(int(np.searchsorted(cum, thr + delta, side="right")), n - 1)
                assert v[lo] <= got[j, c] <= v[hi], (kind, n, rep, c, p, v[lo], got[j, c], v[hi])


# log(1 + e^-|eta|) of well-separated observations, each a small positive term. With
# u = 2^-24 an exponential is within 4 u, the joined factors of 32 observations within
# 2 u per step (ten steps) and their logarithm within 2 u: 32 u of the sum of the
# terms. The rest of the log target is exact (predictors are products of bf16 numbers,
# y eta - max(eta, 0) is zero) but for the final rounding, 2 u of the value.
@pytest.mark.parametrize("form", ["bf16", "tf32", "bf16x1"])
@pytest.mark.parametrize("case", ["8", "12", "14", "17", "mixed", "rare"])
@pytest.mark.parametrize("nobs", [31, 10_000])
def test_glm_well_separated_observations(issm, cuda, form, case, nobs):
    rng = np.random.default_rng(nobs)
    if case == "mixed":
        mag = rng.integers(8 * 8, 25 * 8, size=nobs) / 8.0
    elif case == "rare":
        mag = rng.integers(6 * 8, 14 * 8, size=nobs) / 8.0
    else:
        mag = np.full(nobs, float(case))
    sign = np.ones(nobs) if case in ("8", "17") else -np.ones(nobs) if case == "rare" else rng.choice([-1.0, 1.0], size=nobs)
    X = np.stack([mag * sign, np.zeros(nobs)], axis=1)
    y = (sign > 0).astype(np.float64)
    B = np.array([[1.0, 0.0], [0.5, 0.0], [1.0, 2.0]] * 50, dtype=np.float32)
    prec = {"bf16": issm.native.PREC_BF16, "tf32": issm.native.PREC_TF32, "bf16x1": issm.native.PREC_BF16X1}[form]
    bound = issm.LogisticRegressionTarget(X, y, 10.0).bind(cuda, torch.float32)
    got = bound.evaluate(torch.tensor(B, device=cuda), precision=prec).double().cpu().numpy()
    tail = np.log1p(np.exp(-np.abs(B.astype(np.float64)[:, :1] * X[:, 0]))).sum(1)
    want = -tail - np.log(2 * np.pi * 10.0) - (B.astype(np.float64) ** 2).sum(1) / 20.0
    u = 2.0**-24
    assert np.all(np.abs(got - want) <= 32 * u * tail + 2 * u * np.abs(want))


def test_glm_infinite_predictors(issm, cuda):
    """Predictors that overflow: -inf where every observation disagrees with an
    infinite predictor's side, NaN only where the likelihood is undefined."""
    X = np.array([[3.0e38, 0.0], [3.0e38, 0.0]])
    B = torch.tensor([[4.0, 0.0], [-4.0, 0.0], [float("nan"), 0.0]], device=cuda)
    for prec in (issm.native.PREC_TF32, issm.native.PREC_BF16X1):
        bound = issm.LogisticRegressionTarget(X, np.ones(2), 10.0).bind(cuda, torch.float32)
        got = bound.evaluate(B, precision=prec).cpu().numpy()
        assert np.isnan(got[0]) and got[1] == -np.inf and np.isnan(got[2])


# The SIMT form of the same, in both types: exponentials within 4 u, 64 factors per
# logarithm at 2 u each, the logarithm 2 u, the sums of logarithms error-free (FP32) or one
# rounding per 64 observations and five of the lanes' (FP64): (140 + nobs / 1024) u of
# the sum of the terms; the constant, the prior and the total in the type: 4 u of their sizes.
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("case", ["8", "12", "17", "25", "mixed", "rare"])
@pytest.mark.parametrize("nobs,n", [(31, 40), (10_000, 40), (3000, 5000)])
def test_simt_well_separated_observations(issm, cuda, dtype, case, nobs, n):
    rng = np.random.default_rng(nobs + n)
    if case == "mixed":
        mag = rng.integers(8 * 8, 25 * 8, size=nobs) / 8.0
    elif case == "rare":
        mag = rng.integers(6 * 8, 14 * 8, size=nobs) / 8.0
    else:
        mag = np.full(nobs, float(case))
    sign = -np.ones(nobs) if case in ("8", "17", "rare") else rng.choice([-1.0, 1.0], size=nobs)
    X = np.stack([mag * sign, np.zeros(nobs)], axis=1)
    B = np.zeros((n, 2), dtype=dtype)
    B[:, 0] = np.where(np.arange(n) % 2, 1.0, 0.5)
    B[:, 1] = np.arange(n) % 3
    tdt = torch.float32 if dtype == np.float32 else torch.float64
    bound = issm.LogisticRegressionTarget(X, (sign > 0).astype(np.float64), 10.0).bind(cuda, tdt)
    got = bound.evaluate(torch.tensor(B, device=cuda)).cpu().numpy().astype(np.longdouble)
    B = B.astype(np.longdouble)
    slope, row = np.unique(B[:, 0], return_inverse=True)
    tail = np.log1p(np.exp(-np.abs(slope[:, None] * X[:, 0]))).sum(1)[row]
    const, prior = -np.log(2 * np.longdouble(np.pi) * 10), -(B ** 2).sum(1) / 20
    u = float(np.finfo(dtype).eps) / 2
    bound = (140 + nobs / 1024) * u * tail + 4 * u * (tail + abs(const) + np.abs(prior))
    assert np.all(np.abs(got - (const + prior - tail)) <= bound)


# The smaller terms' sum is a whole number of e^-gap, exact; the exponential, the last
# sum and the logarithm round as in test_f64_log_sum_exp, without its count of terms.
@pytest.mark.parametrize("k", [1025, 4001])
@pytest.mark.parametrize("gap", [37.4, 37.6, 45.0, 59.9, 60.1])
@pytest.mark.parametrize("last", [True, False])
def test_f64_log_sum_exp_of_many_small_terms(issm, cuda, k, gap, last):
    """Many equal terms and one that is `gap` above them, after them or before."""
    db = issm.pack_proposals([issm.FactorGaussian(np.zeros(2), np.eye(2))] * k, cuda)
    x = np.linspace(0.0, 0.5, 20).reshape(10, 2)
    coef = np.full(k, -gap)
    coef[-1 if last else 0] = 0.0
    den = issm.ops.denominator(issm.native.DENOM_FULL, torch.tensor(coef, device=cuda))
    got = issm.ops.mixture_logdensity(db, den, torch.tensor(x, device=cuda)).cpu().numpy()
    xl = x.astype(np.longdouble)
    lq = -np.log(2 * np.longdouble(np.pi)) - 0.5 * (xl * xl).sum(1)
    want = (lq + np.log1p((k - 1) * np.exp(-np.longdouble(gap)))).astype(np.float64)
    # after the maximum each small term meets a sum of at least 1 and may round away: half an ulp of it each
    order = 0.0 if last else 2.0**-53 * k
    assert np.all(np.abs(got - want) <= 2.0**-52 * (16 + 8 * np.abs(lq.astype(np.float64))) + order)


# A forward pass over 8-row blocks: the products L_ik W_kj are sums of at most d / 4 + 8
# rounded terms per thread and two sums across threads, the diagonal block's inverse is
# a substitution of 8 rows: |L W - I| <= (d / 4 + 26) 2^-24 D |L| |W|, D the block diagonal of
# |L_ii| |W_ii|, whatever the condition of the rest.
@pytest.mark.parametrize("d,split", [(16, 8), (24, 16), (40, 16), (48, 32), (63, 16), (64, 16), (64, 32), (64, 40)])
def test_inverse_factor_residual(issm, cuda, d, split):
    """Factors whose lower right part is badly conditioned while its part of the
    inverse stays of order one."""
    rng = np.random.default_rng(d + split)
    L = np.eye(d) + np.tril(0.1 * rng.normal(size=(d, d)), -1)
    low = np.eye(d - split) - np.tril(rng.uniform(0.3, 0.7, size=(d - split, d - split)), -1)
    L[split:, split:] = low
    L[split:, :split] = low @ rng.uniform(-1.0, 1.0, size=(d - split, split)) @ L[:split, :split]
    L = L.astype(np.float32)
    db = issm.pack_proposals([issm.FactorGaussian(np.zeros(d, dtype=np.float32), L)], cuda)
    db.attach_inverse_factors()
    dp = 16 if d <= 16 else 32 if d <= 32 else 64
    loc, fac = torch.empty(d, device=cuda), torch.empty(d, d, device=cuda)
    ln, inv = torch.empty(1, device=cuda), torch.empty(dp, dp, device=cuda)
    L64, fail = L.astype(np.float64), issm.ops.new_failures(cuda)
    issm.ops.fit_factor(torch.zeros(d, device=cuda, dtype=torch.float64), torch.tensor(L64 @ L64.T, device=cuda),
                        torch.eye(d, device=cuda), loc, fac, ln, failures=fail, regularization=0.0, out_inverse=inv)
    pairs = [(L64, db.inverse_factors)]
    if int(fail[0].item()) == 0:  # else L L^T is not positive definite in FP64 and the fit refused it
        pairs.append((fac.double().cpu().numpy().T, inv))
    for factor, inverse in pairs:
        W = inverse.double().cpu().numpy().reshape(dp, dp)[:d, :d]
        D = np.zeros((d, d))
        for b in range(0, d, 8):
            at = slice(b, min(b + 8, d))
            D[at, at] = np.abs(factor[at, at]) @ np.abs(W[at, at])
        bound = (d / 4 + 26) * 2.0**-24 * (D @ (np.abs(factor) @ np.abs(W)))
        assert np.all(np.abs(factor @ W - np.eye(d)) <= bound)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n,d,k,dof", [(100, 3, 8, None), (5000, 16, 8, 5.0), (20_000, 12, 40, None), (700, 24, 8, None),
                                       (333, 33, 20, 4.0), (400_003, 7, 3, None)])
def test_round_in_place(issm, orc, cuda, dtype, n, d, k, dof):
    """Samples written over the normals they are drawn from: the numbers of
    separate arrays."""
    rng = np.random.default_rng(n)
    db, _ = _factor_bank(issm, orc, rng, d, k, dtype, cuda, dof)
    tdt = torch.float32 if dtype == np.float32 else torch.float64
    slots = torch.tensor(rng.integers(0, k, size=n).astype(np.int32), device=cuda)
    normals = torch.tensor(rng.normal(size=n * d).astype(dtype), device=cuda)
    rad = {}
    if dof:
        rad = dict(radial_normals=torch.tensor(rng.normal(size=n * 8).astype(dtype), device=cuda), rn_stride=8,
                   radial_uniforms=torch.tensor(rng.random(size=n * 8).astype(dtype), device=cuda), ru_stride=8)
    den = issm.ops.denominator(issm.native.DENOM_FULL, torch.zeros(k, dtype=tdt, device=cuda))
    db.proposal_ids = torch.arange(1, k + 1, device=cuda)
    want = issm.ops.mis_round(db, den, slots, normals, **rad)
    drawn = issm.ops.draw(db, normals, n, slots=slots, **rad)
    for _ in range(5):
        buf = normals.clone().view(n, d)
        got = issm.ops.mis_round(db, den, slots, buf, samples=buf, **rad)
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    buf = normals.clone().view(n, d)
    assert torch.equal(issm.ops.draw(db, buf, n, slots=slots, out=buf, **rad), drawn)


# A coordinate of a draw is a chain of at most d roundings of its terms and one of the mean:
# (d + 2) eps of the sum of their sizes. Densities as in test_simt_density_shapes.
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("scale", ["factor", "diagonal", "spherical"])
@pytest.mark.parametrize("n,d,k,dof", [(1, 1, 1, None), (127, 4, 3, None), (129, 5, 9, 5.0), (300, 8, 5, None),
                                       (1000, 9, 33, None), (257, 16, 20, 4.0), (500, 17, 3, None), (129, 32, 7, None),
                                       (260, 33, 4, 3.0), (128, 64, 2, None), (90_001, 3, 2, None), (90_001, 13, 5, None)])
def test_simt_scale_kinds(issm, orc, cuda, dtype, scale, n, d, k, dof):
    """Draws from given slots, rounds, densities and appends of every scale kind at
    the edges of the padded dimensions."""
    rng = np.random.default_rng(7 * d + k)
    loc = rng.normal(size=(k, d)).astype(dtype)
    if scale == "factor":
        A = rng.normal(size=(k, d, d))
        sc = np.linalg.cholesky(A @ A.transpose(0, 2, 1) / d + 0.5 * np.eye(d)).astype(dtype)
        dense = sc.astype(np.float64)
        make = issm.FactorGaussian if dof is None else lambda m, s: issm.FactorStudentT(dtype(dof), m, s)
    elif scale == "diagonal":
        sc = (0.5 + rng.random((k, d))).astype(dtype)
        dense = sc[:, :, None].astype(np.float64) * np.eye(d)
        make = issm.DiagonalGaussian if dof is None else lambda m, s: issm.DiagonalStudentT(dtype(dof), m, s)
    else:
        sc = (0.5 + rng.random(k)).astype(dtype)
        dense = sc[:, None, None].astype(np.float64) * np.eye(d)
        make = issm.SphericalGaussian if dof is None else lambda m, s: issm.SphericalStudentT(dtype(dof), m, s)
    db = issm.pack_proposals([make(m, s) for m, s in zip(loc, sc)], cuda)
    ob = orc.BankView(d, orc.GAUSSIAN if dof is None else orc.STUDENT_T,
                      {"factor": orc.SCALE_FACTOR, "diagonal": orc.SCALE_DIAGONAL, "spherical": orc.SCALE_SPHERICAL}[scale],
                      db.locations.double().cpu().numpy(), db.scales.double().cpu().numpy(),
                      db.lognormalizers.double().cpu().numpy(), None if dof is None else db.dofs.double().cpu().numpy(),
                      None if db.range_risk is None else db.range_risk.cpu().numpy())
    tdt = torch.float32 if dtype == np.float32 else torch.float64
    slots = rng.integers(0, k, size=n).astype(np.int32)
    ts = torch.tensor(slots, device=cuda)
    z = rng.normal(size=(n, d)).astype(dtype)
    rad, mult = {}, np.ones((n, 1))
    if dof:
        # uniforms of zero accept the first normal that gives a positive cube: the multiplier is smooth in it
        rn, ru = 0.2 * rng.normal(size=(n, 8)), np.zeros((n, 8))
        rad = dict(radial_normals=torch.tensor(rn.reshape(-1).astype(dtype), device=cuda), rn_stride=8,
                   radial_uniforms=torch.tensor(ru.reshape(-1).astype(dtype), device=cuda), ru_stride=8)
        off = np.float64(dof) / 2 - 1 / 3
        mult = np.sqrt(dof / (2 * off * (1 + rn[:, :1].astype(dtype).astype(np.float64) / (3 * np.sqrt(off))) ** 3))
    x = issm.ops.draw(db, torch.tensor(z.reshape(-1), device=cuda), n, slots=ts, **rad)
    zm = z.astype(np.float64) * mult
    want = loc[slots].astype(np.float64) + np.einsum("irc,ic->ir", dense[slots], zm)
    size = np.abs(loc[slots]).astype(np.float64) + np.einsum("irc,ic->ir", np.abs(dense[slots]), np.abs(zm))
    # a multiplier holds at most ten roundings
    assert np.all(np.abs(x.double().cpu().numpy() - want) <= (d + (14 if dof else 2)) * float(np.finfo(dtype).eps) * size)
    coef = np.log(rng.dirichlet(np.ones(k))).astype(dtype)
    tc = torch.tensor(coef, device=cuda)
    db.proposal_ids = torch.arange(1, k + 1, device=cuda)
    tol = 1e-12 if dtype == np.float64 else 2e-5
    xs = x.double().cpu().numpy().reshape(-1)
    for kind, okind in ((issm.native.DENOM_FULL, orc.DENOM_FULL), (issm.native.DENOM_GENERATING, orc.DENOM_GENERATING)):
        den = issm.ops.denominator(kind, tc)
        rx, lw, _ = issm.ops.mis_round(db, den, ts, torch.tensor(z.reshape(-1), device=cuda), **rad)
        got = issm.ops.mixture_logdensity(db, den, x, slots=ts)
        exp, _, _ = orc.mixture_logdensity(ob, xs, okind, coef.astype(np.float64), slots=slots)
        assert torch.equal(rx, x) and torch.equal(lw, -got)
        assert np.all(np.abs(got.double().cpu().numpy() - exp) <= tol * np.maximum(1.0, np.abs(exp)))
    lognum = torch.tensor(exp.astype(dtype), device=cuda)
    issm.ops.amis_append(db.ref(), k - 1, tc, x, lognum)
    lq, _, _ = orc.mixture_logdensity(ob, xs, orc.DENOM_GENERATING, slots=None, fixed_slot=k - 1)
    expa = np.logaddexp(exp.astype(dtype).astype(np.float64), coef[-1].astype(np.float64) + lq)
    assert np.all(np.abs(lognum.double().cpu().numpy() - expa) <= tol * np.maximum(1.0, np.abs(expa)))


@pytest.mark.parametrize("form", ["bf16", "tf32"])
@pytest.mark.parametrize("d,k", [(64, 5), (33, 9), (16, 40)])
def test_paired_tiles_around_one_per_sm(issm, cuda, form, d, k):
    """As many tiles as SMs and one more, where a CTA begins to take two: the
    rows' numbers do not change."""
    rng = np.random.default_rng(d)
    props = [issm.FactorGaussian(rng.normal(size=d).astype(np.float32),
                                 (np.eye(d) + 0.1 * np.tril(rng.normal(size=(d, d)), -1)).astype(np.float32))
             for _ in range(k)]
    db = issm.pack_proposals(props, cuda)
    db.attach_inverse_factors()
    prec = issm.native.PREC_BF16 if form == "bf16" else issm.native.PREC_TF32
    den = issm.ops.denominator(issm.native.DENOM_FULL, torch.zeros(k, device=cuda))
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    n = 128 * sms
    x = torch.randn(2 * n + 3, d, device=cuda, generator=torch.Generator(device=cuda).manual_seed(2))
    want = issm.ops.mixture_logdensity(db, den, x, precision=prec)
    assert bool(torch.isfinite(want).all())
    for m in (n - 127, n, n + 1):
        assert torch.equal(issm.ops.mixture_logdensity(db, den, x[:m], precision=prec), want[:m])
    issm.ops.check_tensor_core_errors(cuda)


@pytest.mark.parametrize("kind", ["logistic", "linreg"])
@pytest.mark.parametrize("d,nobs,n", [(1, 31, 5), (3, 129, 3), (4, 128, 4863), (6, 2100, 4864), (66, 33, 9)])
def test_f64_regression_of_few_samples(issm, cuda, kind, d, nobs, n):
    """A warp per sample and the line to the tiles, within the bounds of
    test_simt_regression_shapes."""
    test_simt_regression_shapes(issm, cuda, np.float64, kind, d, nobs, n)


# Each exponential holds 1 ulp and its argument's rounding (16 eps at most here), each sum
# n / (512 x 304) + 20 roundings: 64 eps of the sums covers both.
@pytest.mark.parametrize("n", [1, 511, 513, 155_647, 155_649, 700_001])
def test_f64_summary_grid(issm, cuda, n):
    lw = torch.randn(n, device=cuda, dtype=torch.float64, generator=torch.Generator(device=cuda).manual_seed(n)) * 3.0
    got = issm.ops.logweight_summary(lw).cpu().numpy()
    l = lw.cpu().numpy()
    e = np.exp(l - l.max())
    assert got[0] == l.max()
    assert abs(got[1] - e.sum()) <= 64 * 2.0**-52 * e.sum()
    assert abs(got[2] - (e * e).sum()) <= 64 * 2.0**-52 * (e * e).sum()
