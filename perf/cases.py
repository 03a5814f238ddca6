"""Timed cases of the nested MLMC level sampler: the calls that a risk program makes of it, over the
sizes it makes them at.

A case is a dict of plain values; `family` says which public entry point it goes through:

  level    one call Sampler.sample(ell, M), batched streams or the reference's stream layout
  run      a whole continuation MLMC run, Sampler.mlmc_run
  losses   the full-portfolio loss sweep behind the threshold K, Sampler.full_loss
  adjoint  the path-simulated loss with its gradients, Sampler.path_adjoint

Portfolios are synthetic, of the benchmark's distribution: GBM stocks at 100 with r = mu = 0.05
and sigma ~ U[0.1, 0.4], options on uniformly chosen stocks, half calls and half puts, strike
~ U[0.8, 1.2] 100, maturity ~ U[0.25, 2], position ~ N(0, 1).  The threshold K is the 99 % loss
quantile, as in the benchmark, estimated here on 512 outer draws of its own.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nested-risk-mlmc_b200"))
import nmlmc as nm  # noqa: E402

TAU, RATE = nm.TAU_WEEK, 0.05


# ---- the cases ---------------------------------------------------------------------------------
def _level(name, problem, ell, M, **kw):
    """One level call.  problem: shift, reference (the models), portfolio (Black-Scholes) or paths
    (options on the Unbiased method); core: the reference's streams on that many virtual cores."""
    d = dict(name=name, family="level", problem=problem, ell=ell, M=M, N0=32, beta=2, r=1.5, precision="fp32", core=0)
    d.update(kw)
    return d


def listed():
    return [
        # the first call of a run: the reference driver's default M0 = 100, where latency is all
        _level("model_first_call", "reference", 1, 100, beta=4),
        # the reference's model main, to its default tolerance: many rounds of small and middling levels
        dict(name="model_run", family="run", problem="reference", N0=32, beta=4, r=1.5, precision="fp32", tol=1e-3, M0=100),
        # level 0 of a tight tolerance, where a run's outer samples are
        _level("model_level0_large", "shift", 0, 12_000_003),
        # a deep adaptive level, uneven inner counts
        _level("model_level6_adaptive", "shift", 6, 60_001),
        # the same sampler in double precision, the batched run that the FP32 one is checked against
        _level("model_fp64_level", "shift", 3, 20_000, precision="fp64"),
        # the benchmark's large portfolio: importance sub-sampling, delta control variate, adaptive
        _level("portfolio_large_level", "portfolio", 9, 16_000, N0=64, stocks=200, options=1_000_000, sub="importance"),
        # the 20-stock portfolio: uniform sub-sampling, every outer sample at its full count
        _level("portfolio_uniform_level", "portfolio", 6, 20_001, N0=64, r=0.0, stocks=20, options=10_000, sub="uniform"),
        # path-simulated options (randomised Milstein levels) on the batched layout
        _level("portfolio_paths_level", "paths", 3, 3_000, N0=64, stocks=50, options=100_000, sub="importance"),
        # K of the 20-stock portfolio: the 99 % quantile of 1e5 full evaluations
        dict(name="losses_quantile", family="losses", stocks=20, options=10_000, n=100_000, precision="fp32"),
        # loss and gradients of one path-simulated portfolio of 1e5 options
        dict(name="adjoint_single", family="adjoint", portfolios=1, options_lo=100_000, options_hi=100_000, stocks=50,
             M=256, ell=4, pairs=4, precision="fp32"),
        # the reference's own stream layout (the drop-in build, real_t = float), 2048 virtual cores
        _level("dropin_model_level", "reference", 2, 20_000, beta=4, precision="ref32", core=2048),
        # the plain FP64 drop-in on a portfolio: the comparator of the benchmark's headline
        _level("dropin_portfolio_fp64", "portfolio", 2, 6_000, N0=64, precision="fp64", core=2048, stocks=20,
               options=10_000, sub="importance"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["model", "model", "model", "run", "portfolio", "portfolio", "portfolio", "paths", "losses",
                       "losses", "adjoint", "adjoint", "dropin", "dropin_portfolio"])
    if kind == "model":
        ell = rng.randint(0, 7)
        c = _level("", rng.choice(["shift", "reference"]), ell, _log_int(rng, 100, 8_000_000 >> (2 * ell if ell < 5 else 9)),
                   N0=rng.choice([32, 32, 64]), beta=2, r=rng.choice([1.5, 1.5, 0.0]),
                   precision=rng.choice(["fp32", "fp32", "fp64", "ref32"]))
    elif kind == "run":
        c = dict(family="run", problem="reference", N0=32, beta=rng.choice([2, 4]), r=1.5, precision="fp32",
                 tol=round(math.exp(rng.uniform(math.log(8e-4), math.log(8e-3))), 7), M0=rng.choice([100, 1024]))
    elif kind == "portfolio":
        ell = rng.randint(0, 8)
        c = _level("", "portfolio", ell, _log_int(rng, 100, 400_000 >> ell), N0=64, r=rng.choice([1.5, 0.0]),
                   stocks=rng.choice([1, 16, 20, 50, 200]), options=_log_int(rng, 1_000, 300_000),
                   sub=rng.choice(["importance", "uniform"]))
    elif kind == "paths":
        c = _level("", "paths", rng.randint(0, 4), _log_int(rng, 100, 3_000), N0=64, stocks=rng.choice([16, 50]),
                   options=_log_int(rng, 1_000, 100_000), sub=rng.choice(["importance", "uniform"]))
    elif kind == "losses":
        P = _log_int(rng, 1_000, 300_000)
        c = dict(family="losses", stocks=rng.choice([1, 20, 50, 200]), options=P, n=_log_int(rng, 200, 600_000_000 // P),
                 precision=rng.choice(["fp32", "fp32", "fp64"]))
    elif kind == "adjoint":
        n = rng.choice([1, 1, 4, 24])
        hi = _log_int(rng, 2_000, 100_000) // n
        c = dict(family="adjoint", portfolios=n, options_lo=max(50, hi // 4), options_hi=hi, stocks=rng.choice([3, 20, 50]),
                 M=rng.choice([64, 100, 256]), ell=rng.randint(1, 4), pairs=rng.choice([1, 4]),
                 precision=rng.choice(["fp32", "fp32", "fp64"]))
    elif kind == "dropin":
        ell = rng.randint(0, 3)
        c = _level("", rng.choice(["reference", "shift"]), ell, _log_int(rng, 100, 100_000 >> ell), beta=rng.choice([2, 4]),
                   r=rng.choice([1.5, 0.0]), precision=rng.choice(["ref32", "fp64"]), core=rng.choice([64, 2048]))
    else:
        ell = rng.randint(0, 3)
        c = _level("", rng.choice(["portfolio", "portfolio", "paths"]), ell, _log_int(rng, 100, 16_000 >> ell), N0=64,
                   precision=rng.choice(["ref32", "fp64"]), core=2048, stocks=rng.choice([16, 20]),
                   options=_log_int(rng, 500, 20_000), sub=rng.choice(["importance", "uniform"]))
    c.pop("name", None)
    return c


# ---- inputs ------------------------------------------------------------------------------------
def _portfolio(case, seed, options=None, importance=False):
    g = np.random.default_rng([seed, 7])
    Q, P = case["stocks"], options or case["options"]
    pf = dict(S0=np.full(Q, 100.0), mu=np.full(Q, RATE), sigma=0.1 + 0.3 * g.random(Q),
              stock_ind=g.integers(0, Q, P).astype(np.uint32), type=np.where(g.random(P) < 0.5, 1, -1).astype(np.int32),
              strike=100.0 * (0.8 + 0.4 * g.random(P)), maturity=0.25 + 1.75 * g.random(P), w=g.standard_normal(P))
    if importance:                                     # prob ~ |w|, options sorted by it
        order = np.argsort(-np.abs(pf["w"]), kind="stable")
        for k in ("stock_ind", "type", "strike", "maturity", "w"):
            pf[k] = pf[k][order]
    pf["prob"] = np.abs(pf["w"]) if importance else np.ones(P)
    return pf


def _quantile(pf, q, seed, rho=0.0, n=512):
    """Loss quantile of a portfolio over n outer draws of its own (the threshold K)."""
    g = torch.Generator().manual_seed(seed + 3)
    z = torch.randn(n, len(pf["S0"]) + 1, generator=g, dtype=torch.float64).cuda()
    loss = _full_losses(_tensors(pf), _stocks_at_tau(_tensors(pf), z, rho))
    return float(torch.quantile(loss, q))


def _level_seed(seed):
    return (seed * 2654435761 + 12345) & 0x7FFFFFFF


_PREC = dict(fp32=nm.PREC_FP32, fp64=nm.PREC_FP64, ref32=nm.PREC_REF32)
_SUB = dict(importance=nm.SUB_RANDOM, uniform=nm.SUB_UNIFORM)


def _options(case, seed):
    """The portfolio of a level case and the keyword arguments of Sampler.set_portfolio."""
    pf = _portfolio(case, seed, importance=case["sub"] == "importance")
    kw = dict(r=RATE, rho=0.0, tau=TAU, subsample=_SUB[case["sub"]], use_delta_cv=case["sub"] == "importance",
              discount=case["problem"] == "paths" or bool(case["core"]))
    if case["problem"] == "paths":
        kw["methods"] = dict(method=np.full(case["options"], nm.METHOD_UNBIASED, np.int32), dt_h0inv=1, dt_beta=2,
                             dt_prob_expo=-1.5, use_milstein=True, use_antithetic_risk=True)
    kw["max_loss"] = _quantile(pf, 0.99, seed)
    return pf, kw


def _thresholds(seed):
    return 1.0 + 0.01 * (seed % 7), 0.0975 + 0.001 * (seed % 5)     # K of the shift and the reference model


def _sampler(case, seed):
    core = case.get("core", 0)
    return nm.Sampler(0, cores=core or 2048, N0=case["N0"], beta=case["beta"], adaptive_r=case["r"],
                      precision=_PREC[case["precision"]], seed=_level_seed(seed),
                      streams=nm.STREAMS_CORE if core else nm.STREAMS_OUTER)


def prepare(case, seed):
    f = case["family"]
    if f in ("level", "run"):
        s = _sampler(case, seed)
        shift, ref = _thresholds(seed)
        if case["problem"] == "shift":
            s.set_model(nm.MODEL_SHIFT, 0.0, shift)
        elif case["problem"] == "reference":
            s.set_model(nm.MODEL_REFERENCE, 0.02, ref)
        else:
            pf, kw = _options(case, seed)
            s.set_portfolio(pf, **kw)
        return dict(case=case, sampler=s)
    if f == "losses":
        s = nm.Sampler(0, N0=64, precision=_PREC[case["precision"]], seed=_level_seed(seed))
        s.set_portfolio(_portfolio(case, seed), r=RATE, tau=TAU, subsample=nm.SUB_UNIFORM, discount=False)
        return dict(case=case, sampler=s)
    s = nm.Sampler(0, precision=_PREC[case["precision"]], seed=0)
    return dict(case=case, sampler=s, seed=_level_seed(seed), batch=_batch(case, seed))


def _batch(case, seed):
    g = np.random.default_rng([case["portfolios"], case["options_hi"]])     # a case's own sizes, whatever the seed
    sizes = np.exp(g.uniform(math.log(case["options_lo"]), math.log(case["options_hi"]), case["portfolios"]))
    pfs = [_portfolio(case, seed + 100 * k, options=max(1, int(round(P)))) for k, P in enumerate(sizes)]
    return nm.make_batch(pfs, [_quantile(pf, 0.95, seed + k, rho=0.2) for k, pf in enumerate(pfs)], r=RATE, rho=0.2, tau=TAU)


# ---- one pass ----------------------------------------------------------------------------------
def run(state):
    case, s = state["case"], state["sampler"]
    f = case["family"]
    if f == "level":
        r = s.sample(case["ell"], case["M"])
        return {k: r[k] for k in ("fsums", "diffsums", "work", "stats")}
    if f == "run":
        s.reset_streams()                # the same run each time, as a program that reports a seed's result makes it
        r = s.mlmc_run(targetTOL=case["tol"], M0=case["M0"], batched=True)
        out = {k: r[k] for k in ("Eg", "stat_error", "bias_est", "nlevels")}
        for k in ("level_M", "level_fsums", "level_diffsums", "level_work"):      # level tables of one length
            out[k] = np.zeros((24,) + r[k].shape[1:], r[k].dtype)
            out[k][:len(r[k])] = r[k]
        return out
    if f == "losses":
        return s.full_loss(63, 0, case["n"])
    r = s.path_adjoint(state["batch"], ell=case["ell"], pairs=case["pairs"], M=case["M"], seed=state["seed"], loss=True)
    return {k: r[k] for k in ("EL", "P_smooth", "P_hard", "loss", "grad_w_EL", "grad_w_P", "grad_sigma_EL", "grad_sigma_P")}


# ---- the work a pass cannot do without ---------------------------------------------------------
# Operations per unit as the benchmark counts them: a quarter of a counter-generator block, half a
# Box-Muller pair and the sum for one normal (53); half a block, the option draw, Black-Scholes and
# the sum for one sub-sampled option (129); 50 per Black-Scholes evaluation; 58 per antithetic
# path-pair step of the adjoint, 8 more with tangents.
def work(case):
    f = case["family"]
    if f == "run":                       # the estimator's variance p (1 - p) over the tolerance, in level-0 samples
        n = 0.025 / case["tol"] ** 2
        return dict(bytes=4096, flops=n * case["N0"] * 2 * 53)
    if f == "losses":
        return dict(bytes=32 * case["options"] + 8 * case["n"], flops=50 * case["options"] * case["n"])
    if f == "adjoint":
        P = case["portfolios"] * math.sqrt(case["options_lo"] * case["options_hi"])
        steps = P * case["M"] * case["pairs"] * 2 ** case["ell"]
        return dict(bytes=P * (45 + 16) + 8 * case["portfolios"] * case["M"], flops=steps * 66)
    base, top = case["N0"] * max(1, case["beta"] // 2) ** case["ell"], case["N0"] * case["beta"] ** case["ell"]
    # adaptive: one pilot of the fine and the coarse count and the final estimate, at the base count
    inner = top if not 1 < case["r"] < 2 or case["ell"] == 0 else min(3 * base, top)
    ops = {"shift": 53, "reference": 106, "portfolio": 129, "paths": 400}[case["problem"]]
    return dict(bytes=64 + 40 * case.get("options", 0), flops=float(case["M"]) * inner * ops)


# ---- the same results in 64 bits ---------------------------------------------------------------
def _rotl(x, r):
    return (x << r) | ((x >> (64 - r)) & ((1 << r) - 1))


def _i64(v):
    v &= (1 << 64) - 1
    return v - (1 << 64) if v >> 63 else v


def _threefry(c0, c1, k0, k1):
    """Threefry2x64-20 (Salmon et al., SC 2011) on int64 tensors; k0 is a number, the rest broadcast."""
    ks = (torch.tensor(_i64(k0), device=k1.device), k1, _i64(0x1BD11BDAA9FC1A22) ^ _i64(k0) ^ k1)
    x0, x1 = c0 + ks[0] + torch.zeros_like(k1), c1 + ks[1] + torch.zeros_like(c0)
    for rnd in range(20):
        x0 = x0 + x1
        x1 = _rotl(x1, (16, 42, 12, 31, 16, 32, 24, 21)[rnd % 8]) ^ x0
        if rnd % 4 == 3:
            d = rnd // 4 + 1
            x0, x1 = x0 + ks[d % 3], x1 + ks[(d + 1) % 3] + d
    return x0, x1


def _pair(v):
    """Box-Muller of the two 32-bit words of v (uniforms at the cells' middles)."""
    lo, hi = v & 0xFFFFFFFF, (v >> 32) & 0xFFFFFFFF
    a = ((lo ^ 0x80000000) - 0x80000000).double() * 2.0 ** -31 + 2.0 ** -32
    r = torch.sqrt(-2.0 * torch.log(hi.double() * 2.0 ** -32 + 2.0 ** -33))
    return r * torch.sin(math.pi * a), r * torch.cos(math.pi * a)


def _normals(seed, keys, tag, first, n):
    """Normals first .. first + n - 1 (multiples of 4) of phase `tag` for each stream key: [keys, n]."""
    b = torch.arange(first // 4, (first + n + 3) // 4, device=keys.device)
    v0, v1 = _threefry(b[None, :], tag, seed, keys[:, None])
    return torch.stack(_pair(v0) + _pair(v1), -1).reshape(len(keys), -1)[:, :n]


def _tensors(pf):
    d = {k: torch.as_tensor(np.asarray(pf[k], np.float64)).cuda() for k in ("S0", "mu", "sigma", "strike", "maturity", "w", "type")}
    d["s"] = torch.as_tensor(pf["stock_ind"].astype(np.int64)).cuda()
    return d


def _stocks_at_tau(t, z, rho):
    W = math.sqrt(TAU) * (z[:, :1] if len(t["S0"]) == 1 else rho * z[:, :1] + math.sqrt(1 - rho * rho) * z[:, 1:len(t["S0"]) + 1])
    return t["S0"] * torch.exp(t["sigma"] * W + (t["mu"] - t["sigma"] ** 2 / 2) * TAU)


def _cdf(x):
    return 0.5 * torch.special.erfc(-x * math.sqrt(0.5))


def _bs(S, K, T, sg, m):
    sd = sg * torch.sqrt(T)
    d1 = (torch.log(S / K) + (RATE + sg ** 2 / 2) * T) / sd
    return m * S * _cdf(m * d1) - m * K * torch.exp(-RATE * T) * _cdf(m * (d1 - sd)), _cdf(d1) - (m < 0).double()


def _full_losses(t, R, disc=1.0):
    out = torch.empty(len(R), dtype=torch.float64, device=R.device)
    sg = t["sigma"][t["s"]]
    V0 = _bs(t["S0"][t["s"]], t["strike"], t["maturity"], sg, t["type"])[0]
    step = max(1, 16_000_000 // len(V0))
    for a in range(0, len(R), step):
        V = _bs(R[a:a + step][:, t["s"]], t["strike"], t["maturity"] - TAU, sg, t["type"])[0]
        out[a:a + step] = (t["w"] * (V0 - disc * V)).sum(1)
    return out


class _Model:
    def __init__(self, kind, seed, keys, K):
        self.kind, self.seed, self.K = kind, seed, K
        self.Y = _normals(seed, keys, 0, 0, 4)[:, 0]
        self.start = torch.full_like(self.Y, -K)

    def inner(self, keys, at, tag, first, n):
        Y = self.Y[at][:, None]
        if self.kind == "shift":
            return Y + _normals(self.seed, keys, tag, first, n)
        z = _normals(self.seed, keys, tag, 2 * first, 2 * n).reshape(len(keys), n, 2)
        st, s1 = math.sqrt(0.02), math.sqrt(0.98)
        return (st * Y + s1 * z[..., 0]) ** 2 - (st * z[..., 1] + s1 * z[..., 0]) ** 2


class _Uniform:
    """A portfolio of Black-Scholes options with uniform sub-sampling (no control variate)."""

    def __init__(self, case, seed, keys, pf, K):
        self.seed, self.t, self.P = seed, _tensors(pf), case["options"]
        Q = case["stocks"]
        self.R = _stocks_at_tau(self.t, _normals(seed, keys, 0, 0, (Q + 1 + 3) // 4 * 4), 0.0)
        self.V0 = _bs(self.t["S0"][self.t["s"]], self.t["strike"], self.t["maturity"], self.t["sigma"][self.t["s"]], self.t["type"])[0]
        self.start = torch.full((len(keys),), -K, dtype=torch.float64, device=keys.device)

    def inner(self, keys, at, tag, first, n):
        b = torch.arange(first // 2, (first + n) // 2, device=keys.device)
        v = torch.stack(_threefry(b[None, :], tag, self.seed, keys[:, None]), -1).reshape(len(keys), n)
        j = (((v >> 32) & 0xFFFFFFFF) * self.P + (((v & 0xFFFFFFFF) * self.P) >> 32)) >> 32      # floor(v P / 2^64)
        t, s = self.t, self.t["s"][j]
        V = _bs(self.R[at[:, None], s], t["strike"][j], t["maturity"][j] - TAU, t["sigma"][s], t["type"][j])[0]
        return self.P * t["w"][j] * (self.V0[j] - V)


def _sums(P, seed_keys, at, tag, n, block):
    """Per outer sample: the inner values of a phase summed in blocks of `block` samples, and the sum of squares."""
    step = max(1, 8_000_000 // n)
    s1 = torch.empty(len(at), n // block, dtype=torch.float64, device=at.device)
    s2 = torch.empty(len(at), dtype=torch.float64, device=at.device)
    for a in range(0, len(at), step):
        x = P.inner(seed_keys[at[a:a + step]], at[a:a + step], tag, 0, n)
        s1[a:a + step] = x.reshape(len(x), -1, block).sum(2)
        s2[a:a + step] = (x * x).sum(1)
    return s1, s2


def _counts(P, keys, N0, beta, r, ell, tag0):
    top, base = N0 * beta ** ell, N0 * (beta // 2) ** ell
    cnt = torch.full((len(keys),), top, dtype=torch.int64, device=keys.device)
    spent = 0
    if not 1 < r < 2:
        return cnt, spent
    tmp, cur, at, k = top * (9.0 / top) ** (r / 2), base, torch.arange(len(keys), device=keys.device), 0
    while top > 2 * cur and len(at):
        s1, s2 = _sums(P, keys, at, tag0 + k, cur, cur)
        s1 = s1[:, 0]
        spent += cur * len(at)
        var = s2 / (cur - 1) - s1 * s1 / (cur * (cur - 1))
        done = tmp * ((P.start[at] + s1 / cur) ** 2 / var) ** (-r / 2) <= cur
        cnt[at[done]] = cur
        at, cur, k = at[~done], 2 * cur, k + 1
    return cnt, spent


def _exact_level(case, seed):
    ls, M, ell = _level_seed(seed), case["M"], case["ell"]
    fs, ds, work_ = np.zeros(4), np.zeros(4), 0
    if case["problem"] == "portfolio":
        pf, kw = _options(case, seed)
    for a in range(0, M, 2_000_000):
        keys = (ell << 56) + torch.arange(a, min(M, a + 2_000_000), device="cuda")
        if case["problem"] == "portfolio":
            P = _Uniform(case, ls, keys, pf, kw["max_loss"])
        else:
            P = _Model(case["problem"], ls, keys, _thresholds(seed)[case["problem"] == "reference"])
        cf, spent = _counts(P, keys, case["N0"], case["beta"], case["r"], ell, 1)
        cc = torch.zeros_like(cf)
        if ell:
            cc, more = _counts(P, keys, case["N0"], case["beta"], case["r"], ell - 1, 64)
            spent += more
        big, small = torch.maximum(cf, cc), torch.minimum(cf, cc) if ell else cf
        phi_big, phi_small = torch.zeros(len(keys), dtype=torch.float64, device="cuda"), torch.zeros(len(keys), dtype=torch.float64, device="cuda")
        for n, g in torch.unique(torch.stack([big, small], 1), dim=0).tolist():
            at = torch.nonzero((big == n) & (small == g)).flatten()
            s1, _ = _sums(P, keys, at, 128, n, g)
            st = P.start[at]
            phi_big[at] = (st + s1.sum(1) / n >= 0).double()
            phi_small[at] = (st[:, None] + s1 / g >= 0).double().mean(1)
            spent += n * len(at)
        f, c = (phi_big, torch.zeros_like(phi_big)) if not ell else (torch.where(cf > cc, phi_big, phi_small), torch.where(cf > cc, phi_small, phi_big))
        for k in range(4):
            fs[k] += float((f ** (k + 1)).sum())
            ds[k] += float(((f - c) ** (k + 1)).sum()) if ell else 0.0
        work_ += spent
    return dict(fsums=fs, diffsums=ds, work=float(work_), stats=None)


def _exact_losses(case, seed):
    t = _tensors(_portfolio(case, seed))
    out, Q = [], case["stocks"]
    for a in range(0, case["n"], 20_000):
        keys = (63 << 56) + torch.arange(a, min(case["n"], a + 20_000), device="cuda")
        z = _normals(_level_seed(seed), keys, 0, 0, (Q + 1 + 3) // 4 * 4)
        out.append(_full_losses(t, _stocks_at_tau(t, z, 0.0)))
    return torch.cat(out).cpu().numpy()


def _exact_adjoint(case, seed):
    b, ls, M, ell, pairs = _batch(case, seed), _level_seed(seed), case["M"], case["ell"], case["pairs"]
    Q, steps, names = case["stocks"], 2 ** ell, ("EL", "P_smooth", "P_hard", "loss", "grad_w_EL", "grad_w_P", "grad_sigma_EL", "grad_sigma_P")
    out = {k: [] for k in names}
    for p in range(case["portfolios"]):
        o = slice(int(b["option_off"][p]), int(b["option_off"][p + 1]))
        q = slice(int(b["stock_off"][p]), int(b["stock_off"][p + 1]))
        t = _tensors({k: b[k][q if k in ("S0", "mu", "sigma") else o] for k in ("S0", "mu", "sigma", "strike", "maturity", "w", "type", "stock_ind")})
        keys = (ell << 56) + (p << 32) + torch.arange(M, device="cuda")
        z = _normals(ls, keys, 0, 0, (Q + 1 + 3) // 4 * 4)
        R = _stocks_at_tau(t, z, 0.2)
        W = (torch.log(R / t["S0"]) - (t["mu"] - t["sigma"] ** 2 / 2) * TAU) / t["sigma"]
        dR = R * (W - t["sigma"] * TAU)
        P, disc = len(t["w"]), math.exp(-RATE * TAU)
        dl, ds = torch.empty(P, M, dtype=torch.float64, device="cuda"), torch.empty(P, M, dtype=torch.float64, device="cuda")
        nn = pairs * steps
        step = max(1, 16_000_000 // (M * nn))
        for a in range(0, P, step):
            i = torch.arange(a, min(P, a + step), device="cuda")
            s, sg = t["s"][i], t["sigma"][t["s"][i]][:, None]
            K, T, m = t["strike"][i][:, None], t["maturity"][i][:, None], t["type"][i][:, None]
            blk = torch.arange((nn + 3) // 4, device="cuda")
            v0, v1 = _threefry(blk[None, None, :], ((i << 32) | 200)[:, None, None], ls, keys[None, :, None].expand(len(i), M, 1))
            zz = torch.stack(_pair(v0) + _pair(v1), -1).reshape(len(i), M, -1)[..., :nn].reshape(len(i), M, pairs, steps)
            h = ((T - TAU) / steps)[..., None]
            C = dC = 0
            for sign in (1.0, -1.0):
                S = R[:, s].T[..., None].expand(-1, -1, pairs)
                D = dR[:, s].T[..., None].expand(-1, -1, pairs)
                for k in range(steps):
                    dW = sign * torch.sqrt(h) * zz[..., k]
                    g = 1 + RATE * h + sg[..., None] * dW + 0.5 * sg[..., None] ** 2 * (dW * dW - h)
                    D = D * g + S * (dW + sg[..., None] * (dW * dW - h))
                    S = S * g
                x = m[..., None] * (S - K[..., None])
                C = C + 0.5 * torch.clamp(x, min=0).sum(2)
                dC = dC + 0.5 * torch.where(x > 0, m[..., None] * D, 0.0).sum(2)
            S0, m1 = t["S0"][s], t["type"][i]
            V0, _ = _bs(S0, t["strike"][i], t["maturity"][i], sg[:, 0], m1)
            d1 = (torch.log(S0 / K[:, 0]) + (RATE + sg[:, 0] ** 2 / 2) * T[:, 0]) / (sg[:, 0] * torch.sqrt(T[:, 0]))
            vega = S0 * torch.exp(-0.5 * d1 * d1) / math.sqrt(2 * math.pi) * torch.sqrt(T[:, 0])
            f = disc * torch.exp(-RATE * (T - TAU)) / pairs
            dl[i] = V0[:, None] - f * C
            ds[i] = t["w"][i][:, None] * (vega[:, None] - f * dC)
        L, K = (t["w"][:, None] * dl).sum(0), float(b["K"][p])
        delta = 0.01 * abs(K)
        g = torch.sigmoid((L - K) / delta)
        om = g * (1 - g) / (delta * M)
        gs = torch.zeros(Q, M, dtype=torch.float64, device="cuda").index_add_(0, t["s"], ds)
        for k, v in zip(names, (L.mean(), g.mean(), (L > K).double().mean(), L[None], dl.mean(1), dl @ om, gs.mean(1), gs @ om)):
            out[k].append(v.reshape(1) if v.dim() == 0 else v)
    return {k: torch.cat(v).cpu().numpy() for k, v in out.items()}


def exact(case, seed):
    f = case["family"]
    if f == "losses":
        return _exact_losses(case, seed)
    if f == "adjoint":
        return _exact_adjoint(case, seed)
    # None: a whole run (its decisions hang on every digit), the reference's sequential streams (a
    # draw's place depends on all adaptive decisions before it), the alias-table draw and the
    # path-simulated options (tables and per-sample streams of the framework's own)
    if f != "level" or case["core"] or case["problem"] == "paths" or case.get("sub") == "importance":
        return None
    return _exact_level(case, seed)
