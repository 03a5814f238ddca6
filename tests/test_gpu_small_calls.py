"""Calls of few outer samples run as one kernel (a warp per outer sample), larger ones as the
breadth-first launch sequence: the same outer samples must come out of both, record for record
(inner means bit for bit), so a level drawn in small pieces equals the level drawn at once."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

# (kind, precision, N0, beta, r, level, outer samples at once, pieces).  Chunk sums are merged in
# groups of 32 chunks and of 256: N0 = 8 at level 9 reaches 512 chunks of 8, N0 = 4 the shortest
# chunk; r = 0 has no pilots; level 0 is fine-only; 300 stocks exceed the kernel's rows (both calls
# then take the sequence)
CASES = [("shift", "FP32", 32, 2, 1.5, 0, 20_000, (1, 31, 500)), ("shift", "FP32", 32, 2, 1.5, 5, 20_000, (1, 129, 700)),
         ("shift", "FP32", 8, 2, 1.5, 9, 20_000, (3, 200)), ("shift", "FP32", 4, 4, 1.5, 3, 30_000, (100, 5)),
         ("shift", "FP64", 32, 2, 1.5, 7, 10_000, (33, 100)), ("shift", "REF32", 64, 2, 0.0, 4, 5_000, (64, 2)),
         ("ref", "FP32", 32, 4, 1.5, 3, 10_000, (40, 500)), ("ref", "FP64", 16, 2, 1.5, 4, 10_000, (7, 70)),
         ("pf", "FP32", 64, 2, 1.5, 4, 12_000, (50, 300)), ("pf", "FP64", 32, 2, 1.5, 3, 8_000, (50, 11)),
         ("pf", "REF32", 32, 2, 0.0, 2, 8_000, (5, 130)), ("pf1", "FP32", 32, 2, 1.5, 3, 20_000, (9, 90)),
         ("pf300", "FP32", 32, 2, 1.5, 2, 4_000, (10, 10)), ("pfu", "FP32", 64, 2, 0.0, 5, 8_000, (30, 2))]


def _sampler(nm, kind, prec, N0, beta, r):
    s = nm.Sampler(0, N0=N0, beta=beta, adaptive_r=r, precision=getattr(nm, "PREC_" + prec), seed=11)
    s.set_autotune(0)
    if kind == "shift":
        s.set_model(nm.MODEL_SHIFT, 0.0, 1.0)
    elif kind == "ref":
        s.set_model(nm.MODEL_REFERENCE, 0.02, 0.0979)
    else:
        Q = {"pf": 20, "pfu": 7, "pf1": 1, "pf300": 300}[kind]
        imp = kind != "pfu"
        pf = O.synthetic_portfolio(Q, 900, 5, prob="w" if imp else "uniform")
        s.set_portfolio(pf, r=0.05, rho=0.3, max_loss=0.02 * np.abs(pf["w"]).sum(), tau=1 / 52,
                        subsample=nm.SUB_RANDOM if imp else nm.SUB_UNIFORM, use_delta_cv=imp)
    return s


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}-{c[1]}-N{c[2]}-b{c[3]}-r{c[4]}-l{c[5]}")
def test_small_calls_draw_the_same_samples(nm, case):
    kind, prec, N0, beta, r, ell, M, pieces = case
    big = _sampler(nm, kind, prec, N0, beta, r).sample(ell, M, trace=True)["trace"]
    s, at = _sampler(nm, kind, prec, N0, beta, r), 0
    for m in pieces:
        n0 = nm.kernel_launches()
        got = s.sample(ell, m, trace=True)
        if kind != "pf300":
            assert nm.kernel_launches() - n0 == 1                  # one launch
        want = big[at:at + m]
        assert got["trace"].tobytes() == want.tobytes()
        d = want["phi_f"] - (want["phi_c"] if ell else 0)
        tol = 1e-14 if prec == "FP64" else 1e-6                     # the powers of phi are formed in real_t
        for k in range(4):
            np.testing.assert_allclose(got["fsums"][k], (want["phi_f"] ** (k + 1)).sum(), rtol=tol, atol=0)
            np.testing.assert_allclose(got["diffsums"][k], (d ** (k + 1)).sum() if ell else 0, rtol=tol, atol=tol)
        assert got["stats"][1] == m and got["stats"][0] == got["work"]
        at += m


# tiles of the launch sequence hold a power of two of chunks: an N0 of three chunks keeps to it
@pytest.mark.parametrize("prec,r,ell,M,pieces", [("FP32", 1.5, 0, 5_000, (200, 33)), ("FP32", 1.5, 3, 40_000, (300, 7)),
                                                 ("FP64", 0.0, 2, 20_000, (50,))])
def test_counts_of_three_chunks_take_the_sequence(nm, prec, r, ell, M, pieces):
    big = _sampler(nm, "shift", prec, 96, 2, r).sample(ell, M, trace=True)["trace"]
    s, at = _sampler(nm, "shift", prec, 96, 2, r), 0
    for m in pieces:
        n0 = nm.kernel_launches()
        got = s.sample(ell, m, trace=True)["trace"]
        assert nm.kernel_launches() - n0 > 1
        assert got.tobytes() == big[at:at + m].tobytes()
        at += m


# a model's fixed counts of four chunks: one kernel where the outer samples fill the chip, the sequence
# below, the same records
@pytest.mark.parametrize("kind,prec,M,piece", [("ref", "FP32", 9_000, 2_000), ("ref", "FP64", 270_000, 5_000),
                                               ("shift", "REF32", 17_000, 3_000), ("shift", "FP32", 9_000, 5_000)])
def test_fixed_counts_take_the_kernel_that_fills_the_chip(nm, kind, prec, M, piece):
    n0 = nm.kernel_launches()
    big = _sampler(nm, kind, prec, 32, 4, 0.0).sample(1, M, trace=True)["trace"]
    assert nm.kernel_launches() - n0 == 1
    n0 = nm.kernel_launches()
    got = _sampler(nm, kind, prec, 32, 4, 0.0).sample(1, piece, trace=True)["trace"]
    assert nm.kernel_launches() - n0 == (1 if (kind, prec) == ("shift", "FP32") else 2)
    assert got.tobytes() == big[:piece].tobytes()
