"""The adjoint's kept derivatives: outer samples past the kept buffer (1 GiB of derivatives per
call) are recomputed in the pull-back, so a call's gradients come from both kernels.  The loss is
linear in the positions, so sum_i w_i dF/dw_i = sum_m (dF/dL_m) L_m exactly, for F = E[L] and
the smoothed P; the volatilities are checked by central differences along one direction."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(nm, P, K, Q=5, seed=3, dsigma=0.0):
    g = np.random.default_rng(seed)
    pf = dict(S0=np.full(Q, 100.0), mu=np.full(Q, 0.05), sigma=0.1 + 0.3 * g.random(Q) + dsigma,
              stock_ind=g.integers(0, Q, P).astype(np.uint32), type=np.where(g.random(P) < 0.5, 1, -1).astype(np.int32),
              strike=100.0 * (0.8 + 0.4 * g.random(P)), maturity=0.25 + 1.75 * g.random(P), w=g.standard_normal(P) ** 2)
    return nm.make_batch([pf], [K], r=0.05, rho=0.2, tau=1 / 52)


# 2^30 / (16 P) outer samples fit in FP64, 2^30 / (8 P) in FP32: all of the call's, all but one, about
# half; at ell = 0 and 1 several pairs share a block of normals, at ell = 2 none do
@pytest.mark.parametrize("prec,P,M,ell,pairs", [("fp64", 200_000, 335, 0, 1), ("fp64", 200_000, 336, 0, 1),
                                                ("fp64", 150_000, 900, 1, 1), ("fp32", 300_001, 900, 2, 1)])
def test_gradients_across_the_kept_buffer(nm, prec, P, M, ell, pairs):
    s = nm.Sampler(precision=nm.PREC_FP64 if prec == "fp64" else nm.PREC_FP32)
    K = float(np.median(s.path_adjoint(_batch(nm, P, 1.0), ell=ell, pairs=pairs, M=50, seed=9, grads=False, loss=True)["loss"]))
    b = _batch(nm, P, K)
    r = s.path_adjoint(b, ell=ell, pairs=pairs, M=M, seed=9, delta_rel=0.5, loss=True)
    w, L, delta = b["w"], r["loss"][0], 0.5 * abs(K)
    x = 1 / (1 + np.exp(-(L - K) / delta))
    # the same products added in another order: 1e5 terms in double; the FP32 path rounds each
    # w_i l_im once to 24 bits (6e-8 of the sum of magnitudes)
    scale = np.abs(L).sum() / M + (w * np.abs(r["grad_w_EL"])).sum()
    tol = 1e-10 * scale if prec == "fp64" else 1e-7 * scale
    assert abs((w * r["grad_w_EL"]).sum() - L.mean()) <= tol
    assert abs((w * r["grad_w_P"]).sum() - (x * (1 - x) / delta * L).mean()) <= tol / delta
    if prec == "fp64":
        h = 1e-4
        up, dn = (s.path_adjoint(_batch(nm, P, K, dsigma=d), ell=ell, pairs=pairs, M=M, seed=9, delta_rel=0.5, grads=False)
                  for d in (h, -h))
        # second-order in h, plus paths that cross the strike within h: both far below 1e-3 of the slope
        for grad, val in (("grad_sigma_EL", "EL"), ("grad_sigma_P", "P_smooth")):
            cd = (up[val][0] - dn[val][0]) / (2 * h)
            assert abs(r[grad].sum() - cd) <= 1e-3 * np.abs(r[grad]).sum()
