"""exm_autotune after other calls on the same context: it builds the descriptors it times the gather on from the
trajectories that the context holds, leaves the caller's times as they were, and refuses a bank that has not been
analysed."""

import numpy as np
import pytest

import exmarg_b200 as eb
from exmarg_b200 import _lib
from tests.golden_io import Fixture

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ran():
    """(fixture, context): a segment of its bank analysed, then its trajectories made by a stage call"""
    fx = Fixture("config1")
    ctx = _lib.Context(0)
    try:
        bank = fx.b200_bank().clone_for(ctx)
        eb.pe_intrinsic(fx.seg, bank, fx.store, prior=fx.prior_arg, ymin=fx.ymin, n_loud=fx.n_loud,
                        n_random=fx.n_random)
        seg = eb.read_segments(fx.seg)
        bank.trajectories({I: seg["d_" + I][0] for I in "HL"}, {I: seg["sig2_" + I] for I in "HL"})
        yield fx, ctx
    finally:
        ctx.close()


def _tune(ctx, n_loud, n_random):
    try:
        best, ms = ctx.autotune(n_loud, n_random, reps=1)
    finally:
        ctx.set_gather_cfg(0, 150)
    n = len(_lib.GATHER_SHAPES)
    assert 0 <= best < n and np.all(ms[:n + 3] > 0)


@pytest.mark.parametrize("times", ["every time", "of the tuned shape", "of another shape"])
@pytest.mark.parametrize("larger", [False, True])
def test_stage_calls_before_and_after(ran, times, larger):
    fx, ctx = ran
    K, S = (2 * fx.n_loud, 3 * fx.n_random) if larger else (fx.n_loud, fx.n_random)
    if times == "of the tuned shape":
        ctx.select_times(3, K, S)
    elif times == "of another shape":
        ctx.select_times(3, 20, 17)
    nn = len(fx.store.s)
    before = ctx.node_values(nn)
    _tune(ctx, K, S)
    assert np.array_equal(ctx.node_values(nn), before)
    _tune(ctx, 0, 0)
    assert np.array_equal(ctx.node_values(nn), before)


def test_after_uploaded_trajectories_and_another_precision(ran):
    fx, ctx = ran
    rng = np.random.default_rng(1)
    shape = (ctx.nm, ctx.n_time)
    traj = {k: rng.normal(0.0, 1.0, shape).astype(np.float32) for k in ("lqH", "phH", "lqL", "phL")}
    ctx.set_trajectories(traj)
    _tune(ctx, fx.n_loud, fx.n_random)
    ctx.set_filter_precision("fp64")
    _tune(ctx, fx.n_loud, fx.n_random)


def test_a_bank_not_analysed_is_refused(ran):
    fx, ctx = ran
    half = fx.rows.shape[0] // 2
    M, q, chi = (fx.rows[:half, i] for i in range(3))
    bank = eb.MassBank(M, q, chi, fx.seg, "b200", W=fx.W[:half], u=fx.u[:half]).clone_for(ctx)
    eb.prepare(bank, fx.store, fx.prior_arg, fx.ymin)
    with pytest.raises(RuntimeError):
        ctx.autotune(fx.n_loud, fx.n_random, reps=1)
