"""The work that users of this package have it do, as cases that can be timed
and compared: whole sampler calls (static multiple importance sampling, AMIS,
DM-PMC), the tensor-core mixture density and regression likelihood that a
program calls on its own samples, the statistics and resampling of a result,
and the grouped serving loop.

listed() are the cases, draw(rng) gives more of the same ranges, prepare()
makes what a program holds before the call (seeded), run() is one pass through
the public entry points, work() the bytes and operations a pass cannot do
without, exact() the same outputs in 64 bits by plain torch.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """The package directory's name holds a dot, so it is imported by path."""
    if "issm" not in sys.modules:
        pkg = os.path.join(ROOT, "importancesamplers.jl_gb300")
        spec = importlib.util.spec_from_file_location("issm", os.path.join(pkg, "__init__.py"),
                                                      submodule_search_locations=[pkg])
        module = importlib.util.module_from_spec(spec)
        sys.modules["issm"] = module
        spec.loader.exec_module(module)
    return sys.modules["issm"]


DEVICE = "cuda:0"


# ---- the cases ------------------------------------------------------------------
def listed():
    return [
        # static MIS at its full microbenchmark size (4,194,304 samples, 16
        # dimensions, 64 full-covariance Gaussians): one large batch evidence estimate
        _static("static_4m_d16_k64_f32", 16, 64, 4_194_304, "f32", "gaussian", "full"),
        # the smallest call in earnest (the smoke test's size, Float64 as the
        # reference's users run it): launches and host latency
        _static("static_4k_d4_k5_f64", 4, 5, 4096, "f64", "gaussian", "full"),
        # a mid-size Float64 run with heavy-tailed proposals and an odd sample count
        _static("static_100k_d10_k24_t_f64", 10, 24, 100_003, "f64", "student", "full"),
        # the headline AMIS size, 40 rounds of 50,000 samples in 64 dimensions in
        # the BF16 x3 form, on a regression posterior
        _amis("amis_2m_d64_bf16", 64, 40, 50_000, "f32", "bf16", "linreg", 500),
        # a small posterior run as a user's inner loop makes it
        _amis("amis_4k_d5_f32", 5, 4, 1000, "f32", "native", "linreg", 50),
        # the default (plain FP32) form on a ragged mid-size problem
        _amis("amis_80k_d33_f32", 33, 8, 10_007, "f32", "native", "linreg", 500),
        # one population round at the logistic-regression size: 256 factor
        # proposals x 64 samples, p = 32, 10,000 observations
        _dmpmc("dmpmc_256x64_d32", 32, 256, 64, "bf16", 10_000),
        # the regression likelihood of a batch of samples on the tensor cores
        _likelihood("logistic_64k_d32_bf16", 32, 65_536, 10_000, "logistic", "bf16"),
        # re-weighing retained samples under a 40-slot AMIS history
        _density("mixture_1m_d64_k40_bf16", 64, 40, 1_000_003, "bf16"),
        # what is read off a headline-size result: weights, ESS, log Z, mean, resampling
        _posterior("posterior_2m_d64_f32", 64, 2_000_000, "f32", False),
        # the full summary of a mid-size Float64 result, with quantiles and covariance
        _posterior("posterior_100k_d20_f64", 20, 100_003, "f64", True),
        # the serving loop on a burst of mixed posterior requests
        _serve("serve_64", 64, 100_000),
    ]


def _static(name, d, k, n, dtype, family, scheme):
    return dict(name=name, kind="static", d=d, k=k, n=n, dtype=dtype, family=family, scheme=scheme)


def _amis(name, d, rounds, size, dtype, form, target, nobs):
    return dict(name=name, kind="amis", d=d, rounds=rounds, size=size, dtype=dtype, form=form, target=target, nobs=nobs)


def _dmpmc(name, d, k, members, form, nobs):
    return dict(name=name, kind="dmpmc", d=d, k=k, members=members, form=form, nobs=nobs)


def _likelihood(name, d, n, nobs, model, form):
    return dict(name=name, kind="likelihood", d=d, n=n, nobs=nobs, model=model, form=form)


def _density(name, d, k, n, form):
    return dict(name=name, kind="density", d=d, k=k, n=n, form=form)


def _posterior(name, d, n, dtype, summary):
    return dict(name=name, kind="posterior", d=d, n=n, dtype=dtype, summary=summary)


def _serve(name, requests, budget):
    return dict(name=name, kind="serve", requests=requests, budget=budget)


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of the listed ranges: the sizes log-uniform, the dtypes,
    forms and schemes as they come, within the cost of the listed cases."""
    kind = rng.choice(["static", "static", "static", "amis", "amis", "amis", "dmpmc", "likelihood", "density",
                       "posterior", "posterior", "serve"])
    limit = {"f32": 4_194_304 * 64 * 16 * 17, "f64": 300_000 * 24 * 16 * 17}
    while True:
        if kind == "static":
            c = _static(None, rng.randint(2, 64), _log_int(rng, 2, 128), _log_int(rng, 1000, 4_194_304),
                        rng.choice(["f32", "f64"]), rng.choice(["gaussian", "gaussian", "student"]),
                        rng.choice(["full", "full", "random", "standard"]))
            fits = c["n"] * c["k"] * c["d"] * (c["d"] + 1) <= limit[c["dtype"]] and c["n"] * c["d"] <= 67_108_864
        elif kind == "amis":
            form = rng.choice(["native", "bf16", "tf32"])
            dtype = rng.choice(["f32", "f32", "f64"]) if form == "native" else "f32"
            target = rng.choice(["quadratic", "linreg"])
            c = _amis(None, rng.randint(2, 64), rng.randint(2, 40), _log_int(rng, 1000, 50_000), dtype, form, target,
                      _log_int(rng, 50, 2000) if target == "linreg" else 0)
            d, n = c["d"], c["rounds"] * c["size"]
            ops = n * c["rounds"] * d * (d + 1) + n * c["nobs"] * 2 * d
            # enough samples a round for the first fits of a d-dimensional covariance
            fits = c["size"] >= 100 * d and ops <= (3.5e11 if form != "native" else 2e10 if dtype == "f32" else 1.5e9)
        elif kind == "dmpmc":
            c = _dmpmc(None, rng.randint(2, 48), _log_int(rng, 8, 256), rng.randint(8, 64),
                       rng.choice(["native", "bf16", "tf32"]), _log_int(rng, 50, 10_000))
            fits = c["form"] != "native" or c["k"] * c["members"] * c["nobs"] * c["d"] <= 1.5e9
        elif kind == "likelihood":
            c = _likelihood(None, rng.randint(2, 64), _log_int(rng, 1000, 65_536), _log_int(rng, 50, 10_000),
                            rng.choice(["logistic", "linreg"]), rng.choice(["bf16", "tf32", "bf16x1", "native"]))
            fits = c["form"] != "native" or c["n"] * c["nobs"] * c["d"] <= 3e9
        elif kind == "density":
            c = _density(None, rng.randint(2, 64), rng.randint(1, 64), _log_int(rng, 1000, 4_194_304),
                         rng.choice(["bf16", "tf32", "native"]))
            fits = c["n"] * c["k"] <= 40_000_120 and c["n"] * c["d"] <= 134_217_728
            fits = fits and (c["form"] != "native" or c["n"] * c["k"] * c["d"] * (c["d"] + 1) <= 2e10)
        elif kind == "posterior":
            summary = rng.random() < 0.5
            c = _posterior(None, rng.randint(1, 64), _log_int(rng, 1000, 200_000 if summary else 2_000_000),
                           rng.choice(["f32", "f64"]) if not summary else "f64", summary)
            fits = c["d"] * c["n"] <= (2_500_000 if summary else 128_000_000)
        else:
            c = _serve(None, rng.randint(4, 64), _log_int(rng, 2000, 100_000))
            fits = True
        if fits:
            del c["name"]
            return c


# ---- inputs ------------------------------------------------------------------------
def _npdt(case):
    return np.float32 if case.get("dtype", "f32") == "f32" else np.float64


def _tdt(case):
    return torch.float32 if case.get("dtype", "f32") == "f32" else torch.float64


def _seed(case, seed):
    return int(np.random.default_rng([int(seed), 77]).integers(1, 2 ** 62))


def _scale_factors(rng, k, d, floor=0.1):
    """chol(A A^T / d + floor I), A ~ N(0, 1): full covariances of a mixture bank."""
    A = rng.normal(size=(k, d, d))
    return np.linalg.cholesky(A @ A.transpose(0, 2, 1) / d + floor * np.eye(d))


def _bank_arrays(case, seed):
    """Locations, factors (k x d x d), dofs and masses of the case's bank."""
    rng = np.random.default_rng([int(seed), 1])
    d, k, dt = case["d"], case["k"], _npdt(case)
    spread = 2.0 if d <= 16 else 8.0 / math.sqrt(d)
    loc = (spread * rng.normal(size=(k, d))).astype(dt)
    fac = _scale_factors(rng, k, d).astype(dt)
    dofs = rng.choice([3.0, 5.0, 7.5], size=k).astype(dt)
    masses = rng.dirichlet(np.full(k, 4.0))
    return loc, fac, dofs, masses


def _quadratic_problem(case, seed):
    """An unnormalised spherical Gaussian target and a displaced, widened
    Gaussian proposal, as a user starts from a rough mode."""
    rng = np.random.default_rng([int(seed), 2])
    d = case["d"]
    center, divisor = rng.normal(size=d), float(rng.uniform(0.5, 4.0))
    sd, f = math.sqrt(divisor / 2.0), 0.5 / math.sqrt(d)
    return center, divisor, center + f * sd * rng.normal(size=d), (1.0 + f) * sd * np.eye(d)


def _regression_data(rng, nobs, d, logistic):
    X = rng.normal(size=(nobs, d))
    beta = rng.normal(size=d) / (math.sqrt(d) if logistic else 1.0)
    if logistic:
        y = (rng.random(nobs) < 1.0 / (1.0 + np.exp(-(X @ beta)))).astype(np.float64)
    else:
        y = X @ beta + 0.5 * rng.normal(size=nobs)
    return X, y, beta


def _linreg_problem(case, seed):
    """A Bayesian linear regression and the displaced, widened Laplace form of
    its posterior as the initial proposal."""
    rng = np.random.default_rng([int(seed), 3])
    d = case["d"]
    X, y, _ = _regression_data(rng, case["nobs"], d, False)
    A = X.T @ X / 0.25 + np.eye(d)
    mean = np.linalg.solve(A, X.T @ y / 0.25)
    Lp = np.linalg.cholesky(np.linalg.inv(A))
    f = 0.5 / math.sqrt(d)
    return X, y, mean + f * (Lp @ rng.normal(size=d)), (1.0 + f) * Lp


def _posterior_arrays(case, seed):
    g = torch.Generator(device=DEVICE).manual_seed(_seed(case, seed))
    n, d, dt = case["n"], case["d"], _tdt(case)
    scale = torch.rand(d, generator=g, device=DEVICE, dtype=dt) + 0.5
    loc = 2.0 * torch.randn(d, generator=g, device=DEVICE, dtype=dt)
    x = torch.randn(n, d, generator=g, device=DEVICE, dtype=dt) * scale + loc
    lw = torch.randn(n, generator=g, device=DEVICE, dtype=dt) * 1.5 - 12.0
    return x.contiguous(), lw.contiguous()


def _dmpmc_arrays(case, seed):
    """Factor proposals scattered over a logistic posterior's neighbourhood."""
    rng = np.random.default_rng([int(seed), 4])
    d, k = case["d"], case["k"]
    X, y, beta = _regression_data(rng, case["nobs"], d, True)
    loc = (beta + 0.3 * rng.normal(size=(k, d))).astype(np.float32)
    fac = (0.2 * _scale_factors(rng, k, d, 0.3)).astype(np.float32)
    return X, y, loc, fac


def _likelihood_arrays(case, seed):
    rng = np.random.default_rng([int(seed), 5])
    X, y, beta = _regression_data(rng, case["nobs"], case["d"], case["model"] == "logistic")
    x = (beta + 0.3 * rng.normal(size=(case["n"], case["d"]))).astype(np.float32)
    return X, y, x


def _density_arrays(case, seed):
    rng = np.random.default_rng([int(seed), 6])
    d, k = case["d"], case["k"]
    # an adapted history: slots drift about a common centre
    loc = (0.3 * rng.normal(size=(k, d))).astype(np.float32)
    fac = _scale_factors(rng, k, d, 0.5).astype(np.float32)
    logcounts = np.log(rng.integers(1000, 50_000, size=k).astype(np.float64)).astype(np.float32)
    g = torch.Generator(device=DEVICE).manual_seed(_seed(case, seed))
    x = 1.2 * torch.randn(case["n"], d, generator=g, device=DEVICE, dtype=torch.float32)
    return loc, fac, logcounts, x


def _requests(case, seed):
    """The serving mix: d ~ U{2..64}, n_obs log-uniform 50-5000, sample budget
    log-uniform from 1000 over 4 rounds; the initial proposal is the posterior's
    Laplace form displaced and widened by 0.5 / sqrt(d) of its scale."""
    issm = _package()
    rng = np.random.default_rng([case["requests"], case["budget"]])  # the burst's shapes; the data are the seed's
    out = []
    for rid in range(case["requests"]):
        d = int(rng.integers(2, 65))
        nobs = int(math.exp(rng.uniform(math.log(50), math.log(5000))))
        budget = int(math.exp(rng.uniform(math.log(1000), math.log(case["budget"]))))
        X, y, start, fac = _linreg_problem(dict(d=d, nobs=nobs), (int(seed) * 1009 + rid) % (1 << 62))
        p = issm.FactorGaussian(start.astype(np.float32), fac.astype(np.float32))
        target = issm.LinearRegressionTarget(X, y, sigma=0.5, prior_var=1.0)
        out.append(issm.serving.ServeRequest(rid, target, p, rounds=4, round_size=max(budget // 4, 64),
                                             seed=_seed(case, seed) + rid))
    return out


def _form(issm, name):
    n = issm.native
    return {"native": n.PREC_NATIVE, "bf16": n.PREC_BF16, "tf32": n.PREC_TF32, "bf16x1": n.PREC_BF16X1}[name]


def prepare(case, seed):
    issm = _package()
    kind, dt = case["kind"], _npdt(case)
    state = {"kind": kind, "issm": issm}
    if kind == "static":
        loc, fac, dofs, masses = _bank_arrays(case, seed)
        if case["family"] == "gaussian":
            props = [issm.FactorGaussian(m, L) for m, L in zip(loc, fac)]
        else:
            props = [issm.FactorStudentT(v, m, L) for v, m, L in zip(dofs, loc, fac)]
        scheme = {"full": None, "random": issm.RandomMixture(), "standard": issm.StandardMIS()}[case["scheme"]]
        alg = issm.ImportanceSampling(issm.ProposalBank(props, masses), nsamples=case["n"], mis_scheme=scheme)
        state["sampler"] = issm.prepare_sampler(_seed(case, seed), issm.StandardNormalTarget(case["d"]), alg,
                                                device=DEVICE)
    elif kind == "amis":
        if case["target"] == "quadratic":
            center, divisor, start, fac = _quadratic_problem(case, seed)
            target = issm.QuadraticTarget(center, divisor)
        else:
            X, y, start, fac = _linreg_problem(case, seed)
            target = issm.LinearRegressionTarget(X, y, sigma=0.5, prior_var=1.0)
        alg = issm.AMIS(issm.FactorGaussian(start.astype(dt), fac.astype(dt)), rounds=case["rounds"],
                        round_size=case["size"])
        s = issm.prepare_sampler(_seed(case, seed), target, alg, device=DEVICE, precision=_form(issm, case["form"]))
        state["sampler"], state["initial"] = s, tuple(t.clone() for t in s.committed)
    elif kind == "dmpmc":
        X, y, loc, fac = _dmpmc_arrays(case, seed)
        bank = issm.ProposalBank([issm.FactorGaussian(m, L) for m, L in zip(loc, fac)])
        alg = issm.DeterministicMixturePMC(bank, rounds=1, round_size=case["k"] * case["members"],
                                           resampling=issm.LocalResampling())
        s = issm.prepare_sampler(_seed(case, seed), issm.LogisticRegressionTarget(X, y, prior_var=10.0), alg,
                                 device=DEVICE, precision=_form(issm, case["form"]))
        state["sampler"], state["initial"] = s, s.committed_locations
    elif kind == "likelihood":
        X, y, x = _likelihood_arrays(case, seed)
        target = (issm.LogisticRegressionTarget(X, y, prior_var=10.0) if case["model"] == "logistic" else
                  issm.LinearRegressionTarget(X, y, sigma=0.5, prior_var=1.0))
        state["target"] = target.bind(torch.device(DEVICE), torch.float32)
        state["form"] = _form(issm, case["form"])
        state["x"] = torch.from_numpy(x).to(DEVICE)
    elif kind == "density":
        loc, fac, logcounts, x = _density_arrays(case, seed)
        bank = issm.pack_proposals([issm.FactorGaussian(m, L) for m, L in zip(loc, fac)], torch.device(DEVICE))
        bank.attach_inverse_factors()
        coef = torch.from_numpy(logcounts).to(DEVICE)
        state.update(bank=bank, den=issm.ops.denominator(issm.native.DENOM_PREFIX, coef, terms=case["k"]), x=x,
                     slot=case["k"] - 1, form=_form(issm, case["form"]))
    elif kind == "posterior":
        state["x"], state["lw"] = _posterior_arrays(case, seed)
        state["summary"], state["seed"] = case["summary"], _seed(case, seed)
    else:
        state["requests"] = _requests(case, seed)
    return state


# ---- one pass ------------------------------------------------------------------------
def run(state):
    issm, kind = state["issm"], state["kind"]
    if kind == "static":
        r = issm.importance_sample_(state["sampler"])
        return [r.samples, r.logweights, r.provenance["proposal_id"]]
    if kind == "amis":
        s = state["sampler"]
        # every run starts from the same initial proposal, not the last run's
        for dst, src in zip(s.committed, state["initial"]):
            dst.copy_(src)
        r = issm.importance_sample_(s)
        loc, fac, lognorm = issm.current_proposal(s)
        return [r.samples, r.logweights, r.provenance["round"], loc, fac, lognorm]
    if kind == "dmpmc":
        s = state["sampler"]
        s.committed_locations = state["initial"]  # the same population every run
        r = issm.importance_sample_(s)
        return [r.samples, r.logweights, r.provenance["proposal_id"]]
    if kind == "likelihood":
        return state["target"].evaluate(state["x"], precision=state["form"])
    if kind == "density":
        return issm.ops.mixture_logdensity(state["bank"], state["den"], state["x"], fixed_slot=state["slot"],
                                           precision=state["form"])
    if kind == "posterior":
        r = issm.WeightedSamples(state["x"], state["lw"])
        out = [issm.normalized_weights(r), issm.mean(r), float(issm.effective_sample_size(r)),
               float(issm.lognormalizer(r))]
        u = issm.resample(state["seed"], r, count=min(len(r), 200_000))
        out += [u.ancestors, u.samples]
        if state["summary"]:
            out += [issm.quantile(r, [0.05, 0.5, 0.95]), issm.cov(r)]
        return out
    results = issm.serving.GroupedServeLoop(DEVICE).run(state["requests"])
    results.sort(key=lambda r: r.rid)
    if any(r.error is not None for r in results):
        raise RuntimeError("a served run failed")
    # the runs are FP32 runs: their summaries in that type
    return [np.concatenate([r.posterior_mean for r in results]).astype(np.float32),
            torch.tensor([r.logz for r in results]), torch.tensor([r.ess for r in results])]


# ---- what a pass cannot do without ----------------------------------------------------
def work(case):
    kind = case["kind"]
    es = 4 if case.get("dtype", "f32") == "f32" else 8
    if kind == "static":
        n, d, k = case["n"], case["d"], case["k"]
        terms = k if case["scheme"] != "standard" else 1
        return {"bytes": n * (d * es + es + 8) + k * d * d * es, "flops": n * (terms + 1) * d * (d + 1) + 2 * n * d}
    if kind == "amis":
        d, T, n = case["d"], case["rounds"], case["rounds"] * case["size"]
        retained = case["size"] * T * (T + 1) // 2  # samples the T moment fits read
        target = 2 * d * max(case["nobs"], 1)
        return {"bytes": n * (d * es + es + 8) + case["nobs"] * (d + 1) * es,
                "flops": n * T * d * (d + 1) + retained * d * (d + 1) + n * d * (d + 1) + n * target}
    if kind == "dmpmc":
        d, k, n = case["d"], case["k"], case["k"] * case["members"]
        return {"bytes": n * (4 * d + 4 + 8) + k * d * d * 4 + case["nobs"] * (d + 1) * 4,
                "flops": n * (k + 1) * d * (d + 1) + 2 * n * case["nobs"] * d}
    if kind == "likelihood":
        d, n, m = case["d"], case["n"], case["nobs"]
        return {"bytes": 4 * (n * d + n + m * d + m), "flops": 2 * n * m * d}
    if kind == "density":
        d, n, k = case["d"], case["n"], case["k"]
        return {"bytes": 4 * (n * d + n + k * d * d), "flops": n * k * d * (d + 1)}
    if kind == "posterior":
        d, n = case["d"], case["n"]
        count = min(n, 200_000)
        flops = 2 * n * d + 10 * n + (n * d * (d + 1) if case["summary"] else 0)
        return {"bytes": n * d * es + 2 * n * es + count * (2 * d * es + 8), "flops": flops}
    # the mix's means: d = 33, n_obs the log-uniform mean, budget likewise, 4 rounds
    nobs = (5000 - 50) / math.log(100)
    n = (case["budget"] - 1000) / math.log(case["budget"] / 1000)
    d2 = sum(d * d for d in range(2, 65)) / 63
    return {"bytes": case["requests"] * (n * (33 * 4 + 4) + nobs * 34 * 8),
            "flops": case["requests"] * (d2 * nobs + n * d2 * (1 + 1 + 4 + 2.5))}


# ---- 64-bit values ---------------------------------------------------------------------
def _philox(first, count, seed):
    """Philox-4x32-10 blocks first .. first + count - 1 of a stream: 4 int64
    tensors of 32-bit words."""
    mask = 0xFFFFFFFF
    ctr = torch.arange(first, first + count, dtype=torch.int64, device=DEVICE)
    c = [ctr & mask, (ctr >> 32) & mask, torch.zeros_like(ctr), torch.zeros_like(ctr)]
    k0, k1 = seed & mask, (seed >> 32) & mask

    def mul(a, b):
        p = a * b  # wraps mod 2^64: the low and high words are both right
        return (p >> 32) & mask, p & mask

    for _ in range(10):
        h0, l0 = mul(c[0], 0xD2511F53)
        h1, l1 = mul(c[2], 0xCD9E8D57)
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return c


def _words(n, offset, seed, per):
    b0, b1 = offset // per, (offset + n - 1) // per
    return _philox(b0, b1 - b0 + 1, seed), offset - b0 * per


def _uniforms(n, offset, seed, dtype):
    if dtype == "f32":
        w, skip = _words(n, offset, seed, 4)
        u = torch.stack([(v >> 8).double() * 2.0 ** -24 for v in w], 1)
    else:
        w, skip = _words(n, offset, seed, 2)
        u = torch.stack([(((w[1] << 21) | (w[0] >> 11)) & (2 ** 53 - 1)).double(),
                         (((w[3] << 21) | (w[2] >> 11)) & (2 ** 53 - 1)).double()], 1) * 2.0 ** -53
    return u.reshape(-1)[skip:skip + n]


def _normals(n, offset, seed, dtype):
    """Box-Muller pairs in FP64 from the stream's uniforms."""
    if n == 0:
        return torch.empty(0, dtype=torch.float64, device=DEVICE)
    if dtype == "f32":
        w, skip = _words(n, offset, seed, 4)
        pairs = [((w[0] >> 8), (w[1] >> 8)), ((w[2] >> 8), (w[3] >> 8))]
        unit = 2.0 ** -24
    else:
        w, skip = _words(n, offset, seed, 2)
        pairs = [(((w[1] << 21) | (w[0] >> 11)) & (2 ** 53 - 1), ((w[3] << 21) | (w[2] >> 11)) & (2 ** 53 - 1))]
        unit = 2.0 ** -53
    out = []
    for a, b in pairs:
        r = torch.sqrt(-2.0 * torch.log((a.double() + 1.0) * unit))
        t = 2.0 * math.pi * (b.double() * unit)
        out += [r * torch.cos(t), r * torch.sin(t)]
    return torch.stack(out, 1).reshape(-1)[skip:skip + n]


def _t64(a):
    return torch.as_tensor(np.asarray(a, dtype=np.float64), device=DEVICE)


def _radius2(x, loc, fac):
    """|L^-1 (x - loc)|^2 per row, in blocks of rows."""
    out = torch.empty(x.shape[0], dtype=torch.float64, device=DEVICE)
    for i in range(0, x.shape[0], 1 << 18):
        v = (x[i:i + (1 << 18)].double() - loc).T
        out[i:i + (1 << 18)] = torch.linalg.solve_triangular(fac, v, upper=False).square().sum(0)
    return out


def _gaussian(x, loc, fac):
    d = loc.numel()
    return -0.5 * _radius2(x, loc, fac) - 0.5 * d * math.log(2.0 * math.pi) - torch.log(torch.diagonal(fac)).sum()


def _student(x, loc, fac, dof):
    d = loc.numel()
    const = (math.lgamma((dof + d) / 2) - math.lgamma(dof / 2) - d / 2 * math.log(dof * math.pi) -
             float(torch.log(torch.diagonal(fac)).sum()))
    return const - (dof + d) / 2 * torch.log1p(_radius2(x, loc, fac) / dof)


def _mixture(x, locs, facs, coef, dofs=None):
    acc = None
    for k in range(locs.shape[0]):
        lq = coef[k] + (_gaussian(x, locs[k], facs[k]) if dofs is None else _student(x, locs[k], facs[k], float(dofs[k])))
        acc = lq if acc is None else torch.logaddexp(acc, lq)
    return acc


def _regression(x, X, y, model, sigma, prior_var):
    """Log likelihood of every row of x as coefficients, plus the N(0, prior_var I) prior."""
    X, y, b = _t64(X), _t64(y), x.double()
    out = torch.empty(x.shape[0], dtype=torch.float64, device=DEVICE)
    for i in range(0, x.shape[0], 4096):
        eta = b[i:i + 4096] @ X.T
        if model == "logistic":
            out[i:i + 4096] = (y * eta - torch.nn.functional.softplus(eta, threshold=700.0)).sum(1)
        else:
            out[i:i + 4096] = (-0.5 * X.shape[0] * math.log(2.0 * math.pi * sigma ** 2) -
                               (y - eta).square().sum(1) / (2.0 * sigma ** 2))
    d = x.shape[1]
    return out - 0.5 * d * math.log(2.0 * math.pi * prior_var) - b.square().sum(1) / (2.0 * prior_var)


def _radial_multiplier(rn, ru, dofs):
    """sqrt(nu / chi^2_nu) per sample from at most 8 Marsaglia-Tsang attempts."""
    shape = dofs / 2.0
    offset = shape - 1.0 / 3.0  # every dof here is at least 3
    coef = 1.0 / torch.sqrt(offset) / 3.0
    m = torch.full_like(dofs, float("nan"))
    open_ = torch.ones_like(dofs, dtype=torch.bool)
    for a in range(8):
        z, u = rn[:, a], ru[:, a]
        root = 1.0 + coef * z
        cube = root ** 3
        z2 = z * z
        accept = (u < 1.0 - 0.0331 * z2 * z2) | (torch.log(u) < 0.5 * z2 + offset * (1.0 - cube + torch.log(cube)))
        take = open_ & (root > 0) & accept
        m = torch.where(take, torch.sqrt(dofs / (2.0 * offset * cube)), m)
        open_ &= ~take
    return m


def _exact_static(case, seed):
    loc, fac, dofs, masses = _bank_arrays(case, seed)
    n, d, dtype, tdt, sd = case["n"], case["d"], case["dtype"], _tdt(case), _seed(case, seed)
    student = case["family"] == "student"
    mass = masses / masses.max()
    mass = mass / mass.sum()
    order = np.argsort(mass, kind="stable")
    m = mass[order] / mass[order].sum()
    cdf = np.cumsum(m)
    cdf[-1] = 1.0
    logm = np.log(np.diff(np.concatenate([[0.0], cdf])))
    logm -= np.log(np.sum(np.exp(logm)))
    # the assignment is a comparison of numbers of the case's type
    u = _uniforms(n, 0, sd, dtype).to(tdt)
    if case["scheme"] != "random":
        u = (torch.arange(n, device=DEVICE).to(tdt) + u) / n
    slot = torch.searchsorted(torch.as_tensor(cdf.astype(_npdt(case)), device=DEVICE), u, right=False)
    slot = slot.clamp(max=len(order) - 1)
    off = n + 8
    z = _normals(n * d, off, sd, dtype).reshape(n, d)
    off += n * d + 8
    locs, facs, nus = _t64(loc[order]), _t64(fac[order]), _t64(dofs[order])
    if student:
        rn = _normals(n * 8, off, sd, dtype).reshape(n, 8)
        off += n * 8 + 8
        z = z * _radial_multiplier(rn, _uniforms(n * 8, off, sd, dtype).reshape(n, 8), nus[slot])[:, None]
    x = torch.empty(n, d, dtype=torch.float64, device=DEVICE)
    for k in range(len(order)):
        at = torch.nonzero(slot == k).reshape(-1)
        x[at] = locs[k] + z[at] @ facs[k].T
    del z
    logp = -0.5 * d * math.log(2.0 * math.pi) - 0.5 * x.square().sum(1)
    if case["scheme"] == "standard":
        den = torch.empty(n, dtype=torch.float64, device=DEVICE)
        for k in range(len(order)):
            at = torch.nonzero(slot == k).reshape(-1)
            den[at] = _student(x[at], locs[k], facs[k], float(nus[k])) if student else _gaussian(x[at], locs[k], facs[k])
    else:
        den = _mixture(x, locs, facs, logm, nus if student else None)
    return [x, logp - den, torch.as_tensor(order + 1, device=DEVICE)[slot]]


def _exact_amis(case, seed):
    d, T, size, dtype, sd = case["d"], case["rounds"], case["size"], case["dtype"], _seed(case, seed)
    dt = _npdt(case)
    if case["target"] == "quadratic":
        center, divisor, start, fac = _quadratic_problem(case, seed)
        logp = lambda x: -(x - _t64(center)).square().sum(1) / divisor  # noqa: E731
    else:
        X, y, start, fac = _linreg_problem(case, seed)
        logp = lambda x: _regression(x, X, y, "linreg", 0.5, 1.0)  # noqa: E731
    mu, Lk = _t64(start.astype(dt)), _t64(fac.astype(dt))
    total = T * size
    x = torch.empty(total, d, dtype=torch.float64, device=DEVICE)
    lt = torch.empty(total, dtype=torch.float64, device=DEVICE)
    num = torch.empty(total, dtype=torch.float64, device=DEVICE)
    logn = torch.full((T,), math.log(size), dtype=torch.float64, device=DEVICE)
    locs, facs, off = [], [], 0
    ridge = math.sqrt(float(np.finfo(dt).eps))
    for t in range(T):
        old, new = t * size, (t + 1) * size
        x[old:new] = mu + _normals(size * d, off, sd, dtype).reshape(size, d) @ Lk.T
        off += size * d + 8
        locs.append(mu)
        facs.append(Lk)
        lt[old:new] = logp(x[old:new])
        if old:
            num[:old] = torch.logaddexp(num[:old], logn[t] + _gaussian(x[:old], mu, Lk))
        num[old:new] = _mixture(x[old:new], torch.stack(locs), torch.stack(facs), logn)
        lw = lt[:new] - num[:new] + math.log(new)
        w = torch.softmax(lw, 0)
        mean = mu + w @ (x[:new] - mu)
        z = x[:new] - mean
        cov = (z * w[:, None]).T @ z + ridge * float(Lk.square().sum()) / d * torch.eye(d, dtype=torch.float64,
                                                                                       device=DEVICE)
        mu, Lk = mean, torch.linalg.cholesky(cov)
    ids = torch.arange(total, device=DEVICE) // size + 1
    return [x, lw, ids, mu, Lk, float(-0.5 * d * math.log(2.0 * math.pi) - torch.log(torch.diagonal(Lk)).sum())]


def _exact_dmpmc(case, seed):
    X, y, loc, fac = _dmpmc_arrays(case, seed)
    d, k, members, sd = case["d"], case["k"], case["members"], _seed(case, seed)
    n = k * members
    z = _normals(n * d, 0, sd, "f32").reshape(k, members, d)
    locs, facs = _t64(loc), _t64(fac)
    x = (locs[:, None, :] + torch.einsum("kmc,krc->kmr", z, facs)).reshape(n, d)
    coef = [math.log(1.0 / k)] * k
    # 64-bit arithmetic on the FP32 samples that are returned: the likelihood
    # is steep in them
    lp = _regression(x, X, y, "logistic", 0.0, 10.0)
    return [x, lp - _mixture(x, locs, facs, coef), torch.arange(n, device=DEVICE) // members + 1]


def _exact_posterior(case, seed):
    x, lw = _posterior_arrays(case, seed)
    x64, w = x.double(), torch.softmax(lw.double(), 0)
    mean = w @ x64
    logz = float(torch.logsumexp(lw.double(), 0)) - math.log(case["n"])
    out = [w, mean, 1.0 / float(w.square().sum()), logz, None, None]  # resampling is a choice, not a computed number
    if case["summary"]:
        probs, d = [0.05, 0.5, 0.95], case["d"]
        q = torch.empty(len(probs), d, dtype=torch.float64, device=DEVICE)
        for c in range(d):
            v, at = torch.sort(x64[:, c], stable=True)
            cum = torch.cumsum(w[at], 0)
            first = w[at[0]]
            for j, p in enumerate(probs):
                thr = p * (cum[-1] - first) + first
                up = int(torch.searchsorted(cum, thr, right=True).clamp(1, v.numel() - 1))
                q[j, c] = v[up - 1] + (thr - cum[up - 1]) / (cum[up] - cum[up - 1]) * (v[up] - v[up - 1])
        z = x64 - mean
        out += [q, (z * w[:, None]).T @ z]
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "static":
        return _exact_static(case, seed)
    if kind == "amis":
        return _exact_amis(case, seed)
    if kind == "dmpmc":
        return _exact_dmpmc(case, seed)
    if kind == "likelihood":
        X, y, x = _likelihood_arrays(case, seed)
        sigma, pv = (0.0, 10.0) if case["model"] == "logistic" else (0.5, 1.0)
        return _regression(torch.from_numpy(x).to(DEVICE), X, y, case["model"], sigma, pv)
    if kind == "density":
        loc, fac, logcounts, x = _density_arrays(case, seed)
        return _mixture(x, _t64(loc), _t64(fac), _t64(logcounts))
    if kind == "posterior":
        return _exact_posterior(case, seed)
    return None  # a serving burst's runs adapt over four rounds of their own streams
