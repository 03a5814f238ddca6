"""The FP32 full-loss sweep takes outer samples in tiles of 4, 8 or 16 by their number; a sample's
loss is the same whatever tile it falls in, and within the FP32 bound of the FP64 sweep."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


# one stock (rows of one entry), a row padded over the banks, 800 stocks (the most a tile's rows hold)
@pytest.mark.parametrize("Q,P", [(1, 300), (7, 257), (800, 1000)])
def test_losses_do_not_depend_on_the_tile(nm, Q, P):
    pf = O.synthetic_portfolio(Q, P, 6)
    kw = dict(r=0.05, rho=0.2, tau=1 / 52, subsample=nm.SUB_UNIFORM)
    s = nm.Sampler(0, precision=nm.PREC_FP32, seed=4)
    s.set_portfolio(pf, **kw)
    big = s.full_loss(63, 0, 20_003)                                  # tiles of 16, the last one of 3
    for first, n in ((0, 1), (5, 3), (11, 7_999), (2, 8_001), (20_000, 3)):   # of 4 (to 7999) and 8
        np.testing.assert_array_equal(s.full_loss(63, first, n), big[first:first + n])
    s64 = nm.Sampler(0, precision=nm.PREC_FP64, seed=4)
    s64.set_portfolio(pf, **kw)
    # 1e-6 of the terms' magnitudes per option (the FP32 loss's bound), and the FP32 sums of P / 256 terms
    scale = np.abs(pf["w"]).sum() * 300.0
    assert np.abs(big[:4000] - s64.full_loss(63, 0, 4000)).max() <= 1e-6 * scale * (1 + P / 256)
