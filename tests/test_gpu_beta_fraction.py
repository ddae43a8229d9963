"""The fraction of a tap's beta row in the plane gather keeps float32's steps: on a table that is steep in beta, values whose
fraction lies far below one are as exact as the fraction is.  exm_node_values against the float64 oracle."""

import numpy as np
import pytest

import exmarg_b200 as eb
from exmarg_b200 import synth
from oracle import restate

pytestmark = pytest.mark.gpu

STEEP = 1024.0   # of the table, per beta row


def test_small_fractions_keep_their_steps():
    nm, nt, nb = 64, 4096, 100
    rng = np.random.default_rng(3)
    spec = synth.TableSpec(ntau=1, nb=nb, nd=31)
    spec.beta = 0.125 * (np.arange(nb) - 50.0)   # ln|z| / (beta step / 2) exact; s = 1 lies on row 50
    T = np.broadcast_to((STEEP * np.arange(nb, dtype=np.float32))[None, None, :, None], spec.shape)
    s = np.array([1.0, 4.0])                     # rows 50 and 61.09
    store = synth.MemoryStore(spec, s, 3, tables=[np.ascontiguousarray(T)] * 2)
    nu = np.arange(20, 20 + nt // 8 - 19)
    seg = dict(T=1.0, fmin=20.0, fmax=float(nu[-1]), nu=nu)
    bank = eb.MassBank(20.0 + np.arange(nm), np.ones(nm), np.zeros(nm), seg, W=np.zeros((nm, nu.size), np.complex64),
                       u=np.ones(nm))
    # one time a template, its row a fraction of 2^-12 .. 2^-11 above the node's
    lq = (rng.uniform(2.0 ** -12, 2.0 ** -11, (nm, 1)) / 16.0).astype(np.float32) * np.ones((1, bank.n_time), np.float32)
    zero = np.zeros_like(lq)
    traj = dict(lqH=lq, phH=zero, lqL=lq, phL=zero)
    times = (np.full((nm, 1), 5, np.int32), np.zeros((nm, 1), np.float32))
    ctx = eb.Context(0)
    try:
        eb.prepare(bank.clone_for(ctx), store, "volume", 0.1267)
        ctx.set_trajectories(traj)
        ctx.set_times(times)
        ctx.timing(True)
        got = ctx.node_values(2)
        assert ctx.timing(False)["slow_taps"] == 0
    finally:
        ctx.close()
    geo = restate.node_geometry(store.s, store.alpha_lo, store.alpha_hi, bank.u, 0.1267)
    want = restate.node_values(traj, store, geo, [[0, 1]], times)
    assert np.isfinite(want[:2]).all()
    # the fractions lie below 1/8, where a float32 rounds by at most 2^-28: the node's and the sum's; and 2^-21 for the
    # exponential and the float32 sum.  (Steps of 2^-23 would be off by up to 2^-24 STEEP = 6e-5.)
    assert np.abs(got[:2] - want[:2]).max() <= 2 * 2.0 ** -28 * STEEP + 2.0 ** -21
