"""A bounded device wait that runs out: the tensor-core update's pipeline waits given no polls.

The failure is made without faulting or hanging the GPU: caroli_set_wait_limit(ctx, 0) makes
every pipeline wait of tc_update_kernel give up at once, on barriers that have not completed yet.
The kernel then drains the copies and products it issued (those waits keep their own bound),
frees its tensor memory and marks the solve CAROLI_TIMEOUT. The status must reach the caller, a
mixed-precision solve must be recomputed in FP64 (status 105 per block solve) with the oracle's T,
and after the limit is restored the same context must give the oracle's results again.
"""
import numpy as np
import pytest

from systems import bench_system, gradient_bhz, oracle_T
from caroli_gb300 import NestedTwoTerminal, Precision, Region, _native, square
from caroli_gb300.disorder import ScalarPotential

pytestmark = pytest.mark.gpu


def test_wait_limit_timeout_reaches_caller_and_context_recovers():
    sys_ = bench_system("bhz-anderson", 32)  # fronts above 96 variables: the tensor-core update runs
    sigmas = [sys_.self_energies(e) for e in (-0.1, 0.3)]
    ref = [oracle_T(sys_, s) for s in sigmas]
    plan = sys_.plan()
    ctx = plan.ctx
    ctx.set_tensor_cores(True)
    ctx.set_autotune(False)  # the default schedule: fronts above 96 variables on the tensor cores
    try:
        ctx.set_wait_limit(0)
        t, st, _ = sys_.solve_batch(sigmas, [0, 0], Precision.SINGLE)
        assert (st == _native.TIMEOUT).all(), st
        t, st, _ = sys_.solve_batch(sigmas, [0, 0], Precision.MIXED)
        assert (st == _native.OK).all(), st
        _, _, jst = plan.last_job_info()
        assert (np.asarray(jst) == 100 + _native.TIMEOUT).all(), jst
        for tm, r in zip(t, ref):
            assert abs(tm - r) <= 1e-10 * (1 + abs(r)), (tm, r)
    finally:
        ctx.set_wait_limit(-1)
        ctx.set_autotune(True)
    ctx.set_autotune(False)
    t, st, _ = sys_.solve_batch(sigmas, [0, 0], Precision.SINGLE)
    ctx.set_autotune(True)
    assert (st == _native.OK).all(), st
    for ts, r in zip(t, ref):
        assert abs(ts - r) < 1e-2, (ts, r)
    t, st, _ = sys_.solve_batch(sigmas, [0, 0], Precision.MIXED)
    assert (st == _native.OK).all(), st
    _, _, jst = plan.last_job_info()
    assert (np.asarray(jst) == 0).all(), jst
    for tm, r in zip(t, ref):
        assert abs(tm - r) <= 1e-8, (tm, r)


def _f64_device():
    return bench_system("bhz-anderson", 32)  # fronts above 64 variables: the FP64 updates run


def test_f64_wait_limit_reaches_caller_and_context_recovers():
    """The FP64 updates, traces and self-energies formed from lead modes given no polls: every wait gives up on a
    barrier that has not completed, and the kernels drain what they issued."""
    sys_ = _f64_device()
    sigmas = [sys_.self_energies(e) for e in (-0.1, 0.3)]
    ref, st, _ = sys_.solve_batch(sigmas, [0, 0], Precision.DOUBLE)
    assert (st == _native.OK).all(), st
    wire = bench_system("square-anderson", 32)
    wref = wire.transmission_with(wire.self_energies_on_device(0.37))
    ctx = sys_.plan().ctx
    try:
        ctx.set_f64_wait_limit(0)
        _, st, _ = sys_.solve_batch(sigmas, [0, 0], Precision.DOUBLE)
        assert (st == _native.TIMEOUT).all(), st
        with pytest.raises(_native.NativeError, match="wait ran out"):
            wire._slot(wire.self_energies_on_device(0.37))
    finally:
        ctx.set_f64_wait_limit(-1)
    again, st, _ = sys_.solve_batch(sigmas, [0, 0], Precision.DOUBLE)
    assert (st == _native.OK).all(), st
    assert np.array_equal(again, ref)
    assert wire.transmission_with(wire.self_energies_on_device(0.37)) == wref


@pytest.mark.parametrize("length,width", [(2, 9), (2, 60), (2, 150), (24, 40)])
def test_panel_sweep_wait_that_runs_out_is_a_timeout(length, width):
    """Every wait of the panel sweeps given no polls (clusters of 1 to 16 CTAs): the solve is marked TIMEOUT, not
    SINGULAR, and the CTAs only leave when the rows in flight have arrived; the context is as before."""
    clean = square()
    pot = np.random.RandomState(width).uniform(-0.7, 0.7, length * width)
    dev = clean.with_onsite_term(ScalarPotential(pot, width, 1, 1))
    s = NestedTwoTerminal.from_model(dev, clean, Region.cuboid(clean.lattice, [length, width, 0]), 0)
    slot, kept = s._slot(s.self_energies(0.37)), [2 * width]
    ref, st = s.plan().root_green([slot], [0], kept)
    assert st[0] == _native.OK
    ctx = s.plan().ctx
    try:
        ctx.set_f64_wait_limit(0)
        _, st = s.plan().root_green([slot], [0], kept)
        assert st[0] == _native.TIMEOUT
    finally:
        ctx.set_f64_wait_limit(-1)
    again, st = s.plan().root_green([slot], [0], kept)
    assert st[0] == _native.OK
    assert np.array_equal(again[0][0], ref[0][0])


def test_refinement_products_that_time_out_are_reported():
    """The refinement's products given no polls: gradients report TIMEOUT (not a stalled refinement), a mixed
    transmission is recomputed in FP64, which times out as well here; the context is as before afterwards."""
    sys_, derivs = gradient_bhz(24, 12, configs=1)
    sys_.set_parameter_derivatives(derivs)
    sigmas = [sys_.self_energies(e) for e in (-0.1, 0.05)]
    ref = sys_.transmissions_with_grad(sigmas, [0, 0])
    mixed, st, _ = sys_.solve_batch(sigmas, [0, 0], Precision.MIXED)
    assert (ref[1] == _native.OK).all() and (st == _native.OK).all()
    ctx = sys_.plan().ctx
    try:
        ctx.set_f64_wait_limit(0)
        assert (sys_.transmissions_with_grad(sigmas, [0, 0])[1] == _native.TIMEOUT).all()
        _, st, _ = sys_.solve_batch(sigmas, [0, 0], Precision.MIXED)
        assert (st == _native.TIMEOUT).all(), st
    finally:
        ctx.set_f64_wait_limit(-1)
    again = sys_.transmissions_with_grad(sigmas, [0, 0])
    for a, b in zip(again, ref):
        assert np.array_equal(a, b)
    assert np.array_equal(sys_.solve_batch(sigmas, [0, 0], Precision.MIXED)[0], mixed)
