"""Failure handling of the library, made on the host (no GPU fault is provoked):

* a device allocation that fails (nmlmc_inject_alloc_failure) is reported as NMLMC_ERR_NOMEM
  by the call that needed it, and the same context works afterwards with identical results;
* non-finite or non-positive model and portfolio inputs are rejected with NMLMC_ERR_ARG instead
  of turning into phi = 0 inside the kernels.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _model(nm, **kw):
    s = nm.Sampler(N0=32, beta=2, adaptive_r=1.5, precision=nm.PREC_FP32, streams=nm.STREAMS_OUTER, seed=2, **kw)
    s.set_model(nm.MODEL_SHIFT, 0.0, 1.0)
    return s


@pytest.mark.parametrize("after", [0, 3, 8])
def test_allocation_failure_is_reported_and_recoverable(nm, after):
    ref = _model(nm).sample(4, 5000)
    s = _model(nm)
    lib = nm.lib()
    assert lib.nmlmc_inject_alloc_failure(after) == nm.OK
    try:
        with pytest.raises(nm.NmlmcError) as e:
            s.sample(4, 5000)
        assert e.value.status == nm.ERR_NOMEM
    finally:
        lib.nmlmc_inject_alloc_failure(-1)
    s.reset_streams()
    got = s.sample(4, 5000)                 # the context recovers: same streams, same sums
    np.testing.assert_array_equal(got["fsums"], ref["fsums"])
    np.testing.assert_array_equal(got["diffsums"], ref["diffsums"])


def test_allocation_failure_in_a_graph_round(nm):
    s = _model(nm)
    lib = nm.lib()
    lib.nmlmc_inject_alloc_failure(0)
    try:
        with pytest.raises(nm.NmlmcError):
            s.sample_levels([0, 2], [4000, 1000])
    finally:
        lib.nmlmc_inject_alloc_failure(-1)
    s.reset_streams()
    a = s.sample_levels([0, 2], [4000, 1000])
    b = _model(nm).sample_levels([0, 2], [4000, 1000])
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x["fsums"], y["fsums"])


def test_non_finite_inputs_are_rejected(nm):
    s = nm.Sampler(N0=32, beta=2, precision=nm.PREC_FP32, streams=nm.STREAMS_OUTER)
    for tau, K in ((0.0, float("nan")), (float("inf"), 1.0)):
        with pytest.raises(nm.NmlmcError):
            s.set_model(nm.MODEL_SHIFT, tau, K)
    with pytest.raises(nm.NmlmcError):
        s.set_model(nm.MODEL_REFERENCE, 1.5, 0.1)      # sqrt(1 - tau) undefined
    pf = O.synthetic_portfolio(4, 100, 3)
    for key, bad in (("strike", np.nan), ("w", np.inf), ("sigma", 0.0), ("S0", -1.0), ("maturity", np.nan)):
        p = {k: np.array(v, copy=True) for k, v in pf.items()}
        p[key][0] = bad
        with pytest.raises(nm.NmlmcError):
            s.set_portfolio(p, max_loss=1.0)
    with pytest.raises(nm.NmlmcError):
        s.set_portfolio(pf, max_loss=float("nan"))
    s.set_portfolio(pf, max_loss=1.0)                    # the valid portfolio is accepted
    assert s.sample(1, 100)["M"] == 100


@pytest.mark.parametrize("bad", ["stock", "type", "prob", "method"])
def test_a_rejected_portfolio_leaves_the_context_as_it_was(nm, bad):
    """nmlmc_set_portfolio checks everything before it replaces the portfolio in place."""
    pf, other = O.synthetic_portfolio(9, 120, 3), O.synthetic_portfolio(2, 30, 4)
    methods = None
    if bad == "stock":
        other["stock_ind"] = np.array(other["stock_ind"]) + 5
    elif bad == "type":
        other["type"] = np.zeros_like(other["type"])
    elif bad == "prob":
        other["prob"] = np.linspace(1.0, 2.0, 30)               # not falling
    else:
        methods = dict(method=[3] * 30)
    s, ref = _model(nm), _model(nm)
    for x in (s, ref):
        x.set_portfolio(pf, max_loss=1.0)
    with pytest.raises(nm.NmlmcError) as e:
        s.set_portfolio(other, max_loss=5.0, methods=methods)
    assert e.value.status == nm.ERR_ARG
    for ell, M in ((0, 300), (3, 200)):
        a, b = s.sample(ell, M), ref.sample(ell, M)
        np.testing.assert_array_equal(a["fsums"], b["fsums"])
        np.testing.assert_array_equal(a["stats"], b["stats"])
    np.testing.assert_array_equal(s.full_loss(0, 0, 50), ref.full_loss(0, 0, 50))


def _small_batch(nm):
    g = np.random.default_rng(4)
    P, Q = 300, 4
    pf = dict(S0=np.full(Q, 100.0), mu=np.full(Q, 0.05), sigma=0.1 + 0.3 * g.random(Q),
              stock_ind=g.integers(0, Q, P).astype(np.uint32), type=np.where(g.random(P) < 0.5, 1, -1).astype(np.int32),
              strike=100.0 * (0.8 + 0.4 * g.random(P)), maturity=0.25 + 1.75 * g.random(P), w=g.standard_normal(P))
    return nm.make_batch([pf], [1.0], r=0.05, rho=0.2, tau=1 / 52)


@pytest.mark.parametrize("what", ["buffers", "cores", "portfolio", "trace"])
def test_the_adjoints_kept_block_is_given_back_to_other_allocations(nm, what):
    """A context keeps its last nmlmc_path_adjoint's device block; an allocation that fails with it
    in place is tried again without it."""
    lib = nm.lib()

    def call(s):
        if what == "cores":
            s.configure(precision=nm.PREC_REF32, streams=nm.STREAMS_CORE, cores=64)
            s.set_model(nm.MODEL_SHIFT, 0.0, 1.0)
        if what == "portfolio":
            s.set_portfolio(O.synthetic_portfolio(4, 100, 3), max_loss=1.0)
        return s.sample(2, 500, trace=what == "trace")

    want = call(_model(nm))
    s = _model(nm)
    if what == "trace":
        s.sample(2, 500)                        # its buffers are there: the trace's allocation is next
        s.reset_streams()
    adj = s.path_adjoint(_small_batch(nm), ell=2, pairs=1, M=64, seed=3)
    try:
        lib.nmlmc_inject_alloc_failure(0)
        got = call(s)
    finally:
        lib.nmlmc_inject_alloc_failure(-1)
    np.testing.assert_array_equal(got["fsums"], want["fsums"])
    np.testing.assert_array_equal(got["diffsums"], want["diffsums"])
    again = s.path_adjoint(_small_batch(nm), ell=2, pairs=1, M=64, seed=3)
    np.testing.assert_allclose(again["grad_w_EL"], adj["grad_w_EL"], rtol=1e-12, atol=1e-11)


@pytest.mark.parametrize("after", [0, 1])
def test_a_round_without_room_to_overlap_runs_its_levels_in_turn(nm, after):
    """The counters and partial sums of levels that run side by side are optional."""
    lib = nm.lib()
    s, ref = _model(nm), _model(nm)
    s.sample(0, 10)                             # the batch buffers: only the side buffers are left to allocate
    ref.sample(0, 10)
    want = [ref.sample(e, m) for e, m in ((0, 4000), (2, 1000), (5, 300))]
    try:
        lib.nmlmc_inject_alloc_failure(after)
        got = s.sample_levels([0, 2, 5], [4000, 1000, 300])
    finally:
        lib.nmlmc_inject_alloc_failure(-1)
    for x, y in zip(got, want):
        np.testing.assert_array_equal(x["fsums"], y["fsums"])
        np.testing.assert_array_equal(x["diffsums"], y["diffsums"])
        np.testing.assert_array_equal(x["stats"], y["stats"])
    a, b = s.sample_levels([0, 5], [100, 100]), [ref.sample(0, 100), ref.sample(5, 100)]      # with room again
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x["fsums"], y["fsums"])


def test_a_trace_buffer_that_cannot_grow_can_be_used_again(nm):
    lib = nm.lib()
    s, ref = _model(nm), _model(nm)
    want = ref.sample(2, 300, trace=True)
    s.sample(1, 500, trace=True)
    try:
        lib.nmlmc_inject_alloc_failure(0)
        with pytest.raises(nm.NmlmcError) as e:
            s.sample(2, 900, trace=True)
        assert e.value.status == nm.ERR_NOMEM
    finally:
        lib.nmlmc_inject_alloc_failure(-1)
    got = s.sample(2, 300, trace=True)
    assert got["trace"].tobytes() == want["trace"].tobytes()


def test_an_armed_trace_buffer_is_used_by_one_call(nm):
    """A call that fails, or draws nothing, disarms the buffer too: the next one does not write it."""
    s = _model(nm)
    buf = np.zeros(50, nm.TRACE_DTYPE)

    def arm():
        assert nm.lib().nmlmc_set_trace(s.h, buf.ctypes.data, 50) == nm.OK

    arm()
    assert s.sample(2, 0)["M"] == 0
    s.sample(2, 40)
    arm()
    with pytest.raises(nm.NmlmcError):
        s.sample(40, 10)                         # no such level
    s.sample(2, 40)
    arm()
    with pytest.raises(nm.NmlmcError):
        s.sample(2, 60)                          # more samples than the buffer holds
    assert s.sample(2, 60)["M"] == 60
    assert not buf.view(np.uint8).any()
    arm()
    s.sample(2, 40)
    assert buf["count_f"][:40].all() and not buf["count_f"][40:].any()
