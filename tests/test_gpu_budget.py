"""The workspace under a budget: where it does not hold the descriptors of every lag at once, an analysis takes the lags in
several passes, with the results of one pass; and the serving estimate of a worker's workspace covers what one takes."""

import numpy as np
import pytest

import exmarg_b200 as eb
from exmarg_b200 import serve
from tests.golden_io import Fixture

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def stored():
    """the fixtures with a context that holds their tables; its children hold banks and workspaces alone"""
    out = {}
    for name in ("config1", "prodshape"):
        fx = Fixture(name)
        ctx = eb.Context(0)
        eb.prepare(fx.b200_bank().clone_for(ctx), fx.store, fx.prior_arg, fx.ymin)
        out[name] = fx, ctx
    yield out
    for _, ctx in out.values():
        ctx.close()


def _run(stored, name, budget, n_loud, n_random, graph=False):
    """(results, bytes in use, times the gather ran per segment)"""
    fx, parent = stored[name]
    ctx = eb.Context(hbm_budget=budget, share_store_of=parent)
    try:
        ctx.set_graph(graph)
        bank = fx.b200_bank().clone_for(ctx)
        eb.prepare(bank, fx.store, fx.prior_arg, fx.ymin)
        kw = dict(prior=fx.prior_arg, ymin=fx.ymin, n_loud=n_loud, n_random=n_random)
        ctx.timing(True)
        res = eb.pe_intrinsic(fx.seg, bank, fx.store, **kw)
        launches = ctx.timing(False)["gather_launches"] / len(res["ln_b"])
        assert np.array_equal(eb.pe_intrinsic(fx.seg, bank, fx.store, **kw)["ln_lambda"], res["ln_lambda"])
        ctx.autotune(n_loud, n_random, reps=1)
        assert budget == 0 or ctx.bytes <= budget
        return res, ctx.bytes, launches
    finally:
        ctx.close()


@pytest.mark.parametrize("n_loud, n_random", [(1024, 1024), (0, 0)])
@pytest.mark.parametrize("graph", [False, True])
def test_a_smaller_budget_takes_the_lags_in_passes(stored, n_loud, n_random, graph):
    fx, _ = stored["prodshape"]
    want, used, once = _run(stored, "prodshape", 0, n_loud, n_random, graph)
    assert once == 1
    nm, ntau = fx.rows.shape[0], fx.spec.ntau
    walk = n_loud + n_random if n_loud else fx.n_time
    lag = 20 * nm * (walk + 3 * 48)        # descriptors and time indices of one lag
    budget = used - int(0.2 * ntau * lag)
    got, _, passes = _run(stored, "prodshape", budget, n_loud, n_random, graph)
    assert passes > 1
    # the windows of a pass are placed by its own lags: taps change between the float32 windows and the float64 path
    assert np.abs(got["ln_b"] - want["ln_b"]).max() <= 1e-5
    assert np.abs(got["ln_lambda"] - want["ln_lambda"]).max() <= 1e-4


@pytest.mark.parametrize("n_loud, n_random", [(1024, 1024), (100, 60)])
@pytest.mark.parametrize("name", ["config1", "prodshape"])
def test_the_estimate_covers_a_worker(stored, name, n_loud, n_random):
    fx, _ = stored[name]
    _, used, _ = _run(stored, name, 0, n_loud, n_random)
    nm, nf = fx.W.shape
    est = serve.workspace_bytes(nm, fx.n_time, len(fx.store.s), fx.spec.ntau, nf, n_loud + n_random)
    # its margin: 5 % and 64 MiB, room for cuFFT's work area and for residuals of ln|z|, draws of another n_random
    assert used <= est <= 1.05 * (used + nm * (40 * fx.n_time + 8 * 1024)) + (65 << 20)
