"""Batched levels whose N0 is a multiple of 32 but no power of two (96, 160, ...): every inner
sample of a count N0 2^k is drawn and summed.  Against the oracle on the same streams, whose sums
run over the counts as they are: the same counts, phi and level sums, with the tolerances of
test_gpu_parity.py (parity precisions and FP32) and test_gpu_portfolio.py (the FP32 portfolio's).
"""
import ctypes

import numpy as np
import pytest

import oracle as O
from test_gpu_parity import (FLIP_FP32, FLIP_FP64, FLIP_REF32, MARGIN_FP32, MARGIN_FP64, MARGIN_REF32,
                             assert_sums_explained, compare_traces)
from test_gpu_sampler_api import user_lib

pytestmark = pytest.mark.gpu


def _pair(nm, kind, prec, N0, beta, r, seed=9):
    g = nm.Sampler(N0=N0, beta=beta, adaptive_r=r, precision=getattr(nm, "PREC_" + prec), seed=seed)
    o = O.Sampler(O.PREC_REF32 if prec == "REF32" else O.PREC_FP64, O.STREAMS_OUTER, 1, N0, beta, r, True, False, seed)
    g.set_autotune(0)
    if kind in ("shift", "ref"):
        m = (nm.MODEL_SHIFT, 0.0, 1.0) if kind == "shift" else (nm.MODEL_REFERENCE, 0.02, 0.09)
        g.set_model(*m)
        o.set_model(*m)
        return g, o, 1.0
    imp = kind != "uniform"
    pf = O.synthetic_portfolio(5, 200, 4, prob="w" if imp else "uniform")
    kw = dict(r=0.05, rho=0.2, max_loss=1.0, tau=1 / 52, subsample=O.SUB_RANDOM if imp else O.SUB_UNIFORM,
              use_delta_cv=imp)
    if kind == "paths":
        method = [j % 3 for j in range(200)]
        flags = dict(use_coarse_delta_cv=False, use_antithetic_risk=True, use_milstein=True)
        o.set_portfolio_methods(pf, method, **kw, **flags)
        g.set_portfolio(pf, **kw, methods=dict(method=method, **flags))
    else:
        o.set_portfolio(pf, **kw)
        g.set_portfolio(pf, **kw)
    return g, o, float(len(pf["w"]) * np.mean(np.abs(pf["w"]) * (100.0 + pf["strike"])))


# odd factors 3, 5, 9, 11, 33 (a chunk of 4 to 132 samples), 255 (a chunk of 1020); counts of a fraction of
# a warp's chunks, of a tile's and of many tiles
CASES = [("shift", 96, 2, 1.5), ("shift", 160, 4, 0.0), ("shift", 8160, 2, 1.5), ("ref", 96, 4, 1.5), ("ref", 1056, 2, 0.0),
         ("random", 96, 2, 1.5), ("random", 352, 2, 0.0), ("uniform", 288, 2, 1.5), ("paths", 96, 2, 1.5),
         ("paths", 160, 2, 0.0)]
CALLS = [(0, 300), (1, 200), (3, 60), (6, 8)]


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}-N{c[1]}-b{c[2]}-r{c[3]}")
@pytest.mark.parametrize("prec", ["FP64", "REF32", "FP32"])
def test_every_sample_of_an_odd_count_is_drawn(nm, case, prec):
    kind, N0, beta, r = case
    g, o, scale = _pair(nm, kind, prec, N0, beta, r)
    model = kind in ("shift", "ref")
    if model:
        flip = dict(FP64=FLIP_FP64, REF32=FLIP_REF32, FP32=FLIP_FP32)[prec]
    else:                                        # rounding of the losses, scale their sum of magnitudes
        flip = 1e-15 * scale if prec == "FP64" else 2e-6 * scale
    margin = dict(FP64=MARGIN_FP64, REF32=MARGIN_REF32, FP32=MARGIN_FP32)[prec]
    for ell, M in CALLS:
        if N0 * beta ** ell > 70_000:
            continue
        ro = o.sample(ell, M, trace=True, margins=True)
        rg = g.sample(ell, M, trace=True)
        bad = compare_traces(rg["trace"], ro["trace"], flip, max_frac=max(0.02, 2 / M), margins=ro["margins"], margin_bound=margin)
        assert_sums_explained(rg, ro, f32=prec != "FP64")
        if kind != "paths":
            assert rg["stats"][0] == rg["work"]
        if bad == 0:
            assert rg["stats"][0] == ro["stats"][0]


@pytest.mark.parametrize("kind", ["shift", "random", "uniform"])
def test_chunk_lengths_and_variants_of_an_odd_count_agree(nm, kind):
    """Whatever chunk and variant are pinned, the same samples are summed: FP32 traces within the FP32
    bound of each other (the chunk groups the compensated sums differently)."""
    ref = None
    for variant, chunk in ((0, 32), (1, 4), (2, 16), (3, 8), (2, 32)):
        g, _, scale = _pair(nm, kind, "FP32", 96, 2, 0.0)
        g.set_phase_config(3, variant=variant, chunk=chunk)
        t = g.sample(3, 400, trace=True)["trace"]
        if ref is None:
            ref = t
        assert np.abs(t["mean_big"] - ref["mean_big"]).max() <= (FLIP_FP32 if kind == "shift" else 2e-6 * scale)
        assert (t["count_f"] == 768).all() and (t["count_c"] == 384).all()


@pytest.mark.parametrize("ell,r,M", [(0, 1.5, 500), (4, 1.5, 300), (2, 0.0, 300)])
@pytest.mark.parametrize("prec", ["FP32", "FP64"])
def test_other_entry_points_take_an_odd_count(nm, prec, ell, r, M):
    """The allocation-free call and a caller's SAMPLER give the sums of nmlmc_sample."""
    import torch
    g, _, _ = _pair(nm, "shift", prec, 96, 2, r, seed=31)
    want = g.sample(ell, M)
    out = torch.zeros(16, dtype=torch.float64, device="cuda:0")
    rc = nm.lib().nmlmc_sample_level_noalloc(nm.MODEL_SHIFT, 0.0, 1.0, 96, 2, r, 0, getattr(nm, "PREC_" + prec), 31, ell, 0, M,
                                             ctypes.c_void_p(out.data_ptr()), None)
    assert rc == nm.OK
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    np.testing.assert_array_equal(got[0:4], want["fsums"])
    np.testing.assert_array_equal(got[4:8], want["diffsums"])
    assert got[8] == want["work"] == want["stats"][0] == got[9]
    L, dp = user_lib(), ctypes.POINTER(ctypes.c_double)
    assert L.user_shift_init(int(prec == "FP64"), 96, 2, r, 31, 1.0) == nm.OK
    try:
        f, d, w, st = np.zeros(4), np.zeros(4), np.zeros(1), np.zeros(6, np.uint64)
        assert L.user_shift_sample(int(prec == "FP64"), ell, M, f.ctypes.data_as(dp), d.ctypes.data_as(dp),
                                   w.ctypes.data_as(dp), st.ctypes.data_as(ctypes.POINTER(ctypes.c_uint64))) == nm.OK
        np.testing.assert_array_equal(f, want["fsums"])
        np.testing.assert_array_equal(d, want["diffsums"])
        assert w[0] == want["work"] and st[0] == want["stats"][0]
    finally:
        L.user_shift_cleanup()
