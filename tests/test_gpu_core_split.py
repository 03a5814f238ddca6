"""CORE layout (the reference's streams) where its kernel splits or shortens work: outer samples of
one core over several warps at fixed inner counts, outer draws in batches of 64, whole-pair inner
phases and the general ones, and the guide table of the inverse-CDF draw — against the oracle's
sequential restatement, call after call on the same streams."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _same(nm, g, o, calls):
    for ell, M in calls:
        a, b = g.sample(ell, M, trace=True), o.sample(ell, M, trace=True)
        ta, tb = a["trace"], b["trace"]
        # GPU libm against glibc: a phi or a count may differ only at a near-tie, and 300 outer samples
        # of these seeds hold none (the oracle's means and margins are not within 1e-9 of one)
        for f in ("count_f", "count_c", "phi_f", "phi_c", "core", "pilots"):
            np.testing.assert_array_equal(ta[f], tb[f], err_msg=f"{f} at level {ell}")
        np.testing.assert_allclose(ta["mean_big"], tb["mean_big"], rtol=0, atol=1e-6)
        np.testing.assert_allclose(a["fsums"], b["fsums"], rtol=1e-12)
        np.testing.assert_allclose(a["diffsums"], b["diffsums"], rtol=1e-12, atol=1e-12)
        assert a["work"] == b["work"]
        np.testing.assert_array_equal(a["stats"][:6], np.asarray(b["stats"][:6], np.uint64))


# levels with fixed counts (0 and 1, every level at r = 0) split a core's samples over warps: more
# warps than samples, one sample, uneven shares, odd normal counts carried from call to call (N0 = 33:
# no whole pairs; 5: shorter than a warp); adaptive levels between them
@pytest.mark.parametrize("kind", [O.MODEL_SHIFT, O.MODEL_REFERENCE])
@pytest.mark.parametrize("cores,N0,beta,r,anti", [(1, 32, 2, 1.5, True), (3, 33, 2, 1.5, True), (7, 5, 4, 0.0, True),
                                                  (64, 64, 2, 0.0, False), (2048, 32, 4, 1.5, True)])
def test_split_levels_match_the_oracle(nm, kind, cores, N0, beta, r, anti):
    for prec, oprec in ((nm.PREC_FP64, O.PREC_FP64), (nm.PREC_REF32, O.PREC_REF32)):
        g = nm.Sampler(cores=cores, N0=N0, beta=beta, adaptive_r=r, antithetic=anti, precision=prec,
                       streams=nm.STREAMS_CORE, seed=5)
        o = O.Sampler(oprec, O.STREAMS_CORE, cores, N0, beta, r, anti, False, 5)
        for s in (g, o):
            s.set_model(kind, 0.02, 1.0 if kind == O.MODEL_SHIFT else 0.0979)
        _same(nm, g, o, [(0, 1), (0, 143), (1, 131), (2, 65), (0, 300), (1, 1), (0, 2)])


# importance draws: equal, geometric (buckets with many options, empty buckets) and one dominating
# probability, down to one option; fixed counts (one option has no spread for the adaptive rule to see)
@pytest.mark.parametrize("P,shape", [(1, "one"), (2, "geo"), (3, "one"), (100, "equal"), (257, "geo"), (3000, "one"), (4096, "abs")])
def test_guided_cdf_draws_match_the_oracle(nm, P, shape):
    pf = O.synthetic_portfolio(3, P, 4)
    k = np.arange(P)
    pf["prob"] = {"one": np.where(k == 0, 1.0, 1e-4), "geo": 0.97 ** np.minimum(k, 200), "equal": np.ones(P),
                  "abs": np.sort(np.abs(np.random.default_rng(1).standard_normal(P)))[::-1] + 1e-6}[shape]
    kw = dict(r=0.05, rho=0.3, max_loss=1.0, tau=1 / 52, subsample=O.SUB_RANDOM, use_delta_cv=True)
    for prec, oprec in ((nm.PREC_FP64, O.PREC_FP64), (nm.PREC_REF32, O.PREC_REF32)):
        g = nm.Sampler(cores=4, N0=32, beta=2, adaptive_r=0.0, precision=prec, streams=nm.STREAMS_CORE, seed=8)
        o = O.Sampler(oprec, O.STREAMS_CORE, 4, 32, 2, 0.0, True, False, 8)
        g.set_portfolio(pf, **kw)
        o.set_portfolio(pf, **kw)
        for ell, M in ((0, 60), (2, 25)):
            a, b = g.sample(ell, M, trace=True)["trace"], o.sample(ell, M, trace=True)["trace"]
            np.testing.assert_array_equal(a["count_f"], b["count_f"])
            # another option anywhere moves an inner mean by far more than the libm difference
            scale = np.abs(b["mean_big"]).max()
            np.testing.assert_allclose(a["mean_big"], b["mean_big"], rtol=0, atol=(1e-9 if prec == nm.PREC_FP64 else 1e-4) * scale)
