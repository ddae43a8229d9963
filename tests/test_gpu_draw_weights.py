"""The importance weight of the random draws in the plane gather: a draw keeps its weight whatever its phase (equal
phases in both detectors give it a plane weight of exactly zero) and whatever log weight the caller gives, on the staged
windows and on the exact path.
exm_node_values against the float64 oracle on the same float32 trajectories and times."""

import numpy as np
import pytest

import exmarg_b200 as eb
from oracle import restate
from tests.test_gpu_gather_edges import NT, _case

pytestmark = pytest.mark.gpu

NODES = 4


def _node_values(store, bank, traj, times):
    """(node values, taps on the exact path)"""
    ctx = eb.Context(0)
    try:
        eb.prepare(bank.clone_for(ctx), store, "volume", 0.1267)
        ctx.set_trajectories(traj)
        ctx.set_times(times)
        ctx.timing(True)
        got = ctx.node_values(NODES)
        return got, ctx.timing(False)["slow_taps"]
    finally:
        ctx.close()


def _tolerance(store):
    # as for the gather's edge sizes: a dozen roundings of 2^-23 of a tap's interpolation term, and chains of at most 64
    # float32 additions of relative error 2^-24 each
    step = max(np.abs(np.diff(T, axis=a)).max() for T in store.tables for a in (1, 2, 3))
    return 12 * 2.0 ** -23 * max(1.0, 3.0 * step) + 64 * 2.0 ** -24


def _check(got, want, tol):
    assert np.array_equal(np.isfinite(got), np.isfinite(want)) and np.isfinite(want).any()
    fin = np.isfinite(want)
    assert np.abs(got[fin] - want[fin]).max() <= tol


@pytest.mark.parametrize("dtype", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("phases", ["constant", "zero lag"])
@pytest.mark.parametrize("path", ["windows", "exact"])
def test_a_draw_of_equal_phases_keeps_its_weight(dtype, phases, path):
    nm, walk = 40, 300
    store, bank, traj, rng = _case(nm, 5, 200, 219, NODES, 11)
    if phases == "constant":     # every tap at a difference of zero
        traj["phH"][:] = traj["phL"][:] = np.float32(0.7)
    else:                        # the taps of lag 0
        traj["phH"][:] = traj["phL"]
    if path == "exact":          # ln|z_L| over more rows than the windows have, beyond the table at both ends
        traj["lqL"] += rng.uniform(-14.0, 14.0, traj["lqL"].shape).astype(np.float32)
    sel = np.sort(np.stack([rng.choice(NT, walk, replace=False) for _ in range(nm)]), axis=1).astype(np.int32)
    # draws of weight e^3 = 20 beside loud times: without the weight the values move by about one
    lw = np.where(rng.random(sel.shape) < 0.5, np.float32(3.0), np.float32(0.0))
    store_d = eb.with_table_dtype(store, dtype) if dtype != "f32" else store
    got, slow = _node_values(store_d, bank, traj, (sel, lw))
    taps = 5 * walk * nm * NODES
    assert slow > 0.1 * taps if path == "exact" else slow < 0.05 * taps
    store.tables = [eb.quantize_table(T, dtype)[0] for T in store.tables]
    geo = restate.node_geometry(store.s, store.alpha_lo, store.alpha_hi, bank.u, 0.1267)
    want = restate.node_values(traj, store, geo, [list(range(NODES))], (sel, lw))
    _check(got, want, _tolerance(store))


@pytest.mark.parametrize("lw", [-200.0, -90.0, -61.0, 60.0, 61.0, 95.0, 200.0])
@pytest.mark.parametrize("draws", ["all", "half"])
@pytest.mark.parametrize("dtype, path", [("f32", "windows"), ("f32", "exact"), ("f16", "windows")])
def test_any_log_weight(lw, draws, dtype, path):
    nm, walk = 40, 300
    store, bank, traj, rng = _case(nm, 5, 200, 219, NODES, 12)
    if path == "exact":
        traj["lqL"] += rng.uniform(-14.0, 14.0, traj["lqL"].shape).astype(np.float32)
    sel = np.sort(np.stack([rng.choice(NT, walk, replace=False) for _ in range(nm)]), axis=1).astype(np.int32)
    drawn = np.ones(sel.shape, bool) if draws == "all" else rng.random(sel.shape) < 0.5
    times = (sel, np.where(drawn, np.float32(lw), np.float32(0.0)))
    store_d = eb.with_table_dtype(store, dtype) if dtype != "f32" else store
    got, _ = _node_values(store_d, bank, traj, times)
    store.tables = [eb.quantize_table(T, dtype)[0] for T in store.tables]
    geo = restate.node_geometry(store.s, store.alpha_lo, store.alpha_hi, bank.u, 0.1267)
    want = restate.node_values(traj, store, geo, [list(range(NODES))], times)
    # and two roundings of a float32 sum of the weight and the interpolation term
    _check(got, want, _tolerance(store) + 2 * 2.0 ** -24 * (abs(lw) + 10.0))
