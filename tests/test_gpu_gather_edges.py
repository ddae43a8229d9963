"""The plane gather and its tap build at the sizes where their splits change: runs shorter than a group of four taps,
one template (adjacent runs of different plane pairs), chunks of one, two and four groups per lane, several template
chunks and parts of the plane pairs per node, windows taller than the table, lags that are no multiple of a warp, walks
longer than the scatter's cache, boundary points.  exm_node_values against the float64 oracle on the same float32
trajectories and times."""

import numpy as np
import pytest

import exmarg_b200 as eb
from exmarg_b200 import synth
from oracle import restate

pytestmark = pytest.mark.gpu

NT = 4096


def _case(nm, ntau, nb, nd, nodes, seed):
    rng = np.random.default_rng(seed)
    spec = synth.TableSpec(ntau=ntau, nb=nb, nd=nd)
    # s / u around the amplitude axis' lower end, so that boundary points occur as well as interior ones
    s = np.geomspace(0.03, 40.0, nodes)
    # gentle tables (steps below 0.2), so that the tolerance is far below the weight of a single tap
    r, c, b, d = np.meshgrid(np.arange(ntau), np.arange(49), np.arange(nb), np.arange(nd), indexing="ij", sparse=True)
    tables = [(3.0 * np.sin(0.05 * b + 0.3 * k) + 2.0 * np.cos(0.04 * d + 0.1 * r) * np.cos(0.06 * c) - 0.5 * k
               + 0.02 * rng.standard_normal((ntau, 49, nb, nd))).astype(np.float32) for k in range(nodes)]
    store = synth.MemoryStore(spec, s, 11, tables=tables)
    u = np.exp(rng.uniform(0.0, 0.8, nm))
    nu = np.arange(20, 20 + NT // 8 - 19)
    seg = dict(T=1.0, fmin=20.0, fmax=float(nu[-1]), nu=nu)
    W = np.zeros((nm, nu.size), np.complex64)
    bank = eb.MassBank(20.0 + np.arange(nm), np.ones(nm), np.zeros(nm), seg, W=W, u=u)
    assert bank.n_time == NT
    z = rng.normal(size=(4, nm, NT)) * 1.2
    amp = np.exp(rng.normal(0.0, 0.6, (nm, 1)))
    lq = [np.log(np.hypot(z[2 * i], z[2 * i + 1]) * amp + 1e-6).astype(np.float32) for i in range(2)]
    ph = [np.arctan2(z[2 * i + 1], z[2 * i]).astype(np.float32) for i in range(2)]
    return store, bank, dict(lqH=lq[0], phH=ph[0], lqL=lq[1], phL=ph[1]), rng


@pytest.mark.parametrize("nm,ntau,nb,nd,nodes,walk,dtype", [
    (1, 3, 100, 109, 4, 40, "f32"),        # one template: neighbouring runs differ in the plane pair alone
    (2, 1, 40, 31, 3, 3, "f32"),           # fewer taps than plane pairs; a table lower than the windows
    (5, 33, 100, 109, 3, 129, "f32"),      # one lag beyond a warp
    (64, 5, 200, 219, 6, 1024, "f32"),     # several groups per lane
    (300, 3, 100, 219, 5, 257, "bf16"),    # 16-bit windows, more templates than a block's least
    (700, 1, 100, 109, 3, 2048, "f16"),    # chunks of four groups per lane
    (3, 3, 100, 109, 4, 0, "f32"),         # every time: longer than the scatter's cache
])
def test_node_values_at_the_edges(nm, ntau, nb, nd, nodes, walk, dtype):
    store, bank, traj, rng = _case(nm, ntau, nb, nd, nodes, 7 * nm + ntau)
    times = None
    if walk:
        sel = np.sort(np.stack([rng.choice(NT, walk, replace=False) for _ in range(nm)]), axis=1).astype(np.int32)
        lw = np.where(rng.random(sel.shape) < 0.5, np.float32(1.75), np.float32(0.0))
        times = (sel, lw)
    store_d = eb.with_table_dtype(store, dtype) if dtype != "f32" else store
    ctx = eb.Context(0)
    try:
        own = bank.clone_for(ctx)
        eb.prepare(own, store_d, "volume", 0.1267)
        ctx.set_trajectories(traj)
        ctx.set_times(times)
        got = ctx.node_values(nodes)
        again = ctx.node_values(nodes)
    finally:
        ctx.close()
    store.tables = [eb.quantize_table(T, dtype)[0] for T in store.tables]
    geo = restate.node_geometry(store.s, store.alpha_lo, store.alpha_hi, bank.u, 0.1267)
    want = restate.node_values(traj, store, geo, [list(range(nodes))], times)
    assert np.array_equal(np.isfinite(got), np.isfinite(want)) and np.isfinite(want).any()
    assert np.isfinite(want[nodes]).any()
    fin = np.isfinite(want)
    # a tap is the stored value plus a float32 interpolation term: its corners differ by at most the table's largest
    # step along each of three axes, and a dozen roundings of 2^-23 of that; the sums of exponentials are chains of
    # at most 64 float32 additions (a lane's taps, the lanes, the pairs) of relative error 2^-24 each
    step = max(np.abs(np.diff(T, axis=a)).max() for T in store.tables for a in (1, 2, 3))
    assert np.abs(got[fin] - want[fin]).max() <= 12 * 2.0 ** -23 * max(1.0, 3.0 * step) + 64 * 2.0 ** -24
    assert np.array_equal(got, again)   # the order of the sums does not depend on the run
