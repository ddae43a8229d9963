"""Measured cases: the work a user of exmarg_b200 has it do, through its public entry points.

Kinds of case
* pe            pe_intrinsic on one or a few H1/L1 segments with a resident store and a kept bank: the analysis itself
                (matched filter, time selection, table gather, node and distance log-sum-exp, ln B).
* redshift      pe_redshift: the same stages for an equal-mass bank, then the (m1, z) surface, returned whole.
* gather        Context.gather, the gather_cpu / gather_gpu contract, on trajectories and times the program holds.
* trajectories  MassBank.trajectories: one segment's matched filter, the trajectories on the host.
* wtable        wtable.w_table: stage 1 of the offline table build over a few sky pixels.
* tables        Context.k_edges and tables.bd_tables: stages 2 and 3 for one node's W.

Stores are the seeded synthetic tables of the production geometry (generated on the device), banks seeded Latin
hypercubes of TaylorF2 templates; both are kept by the program for all of its segments, so they do not depend on a
case's seed.  Segments (noise and injections), W tables and grids' data do.

The analysis returns float64 arrays whose values carry single precision: tables, trajectories and interpolation are
float32 by design (the documented accuracy of ln Lambda and ln B is 1e-5).  A program keeps such results in float32,
and so do the cases; the float64 gather contract is returned as it comes.
"""

import math

import numpy as np
import torch

import exmarg_b200 as eb
from exmarg_b200 import synth, tables, wtable

TABLE_SEED, BANK_SEED = 2026, 11
YMIN = 0.1267
NPHI, D0 = 96, 10410.0


# ----------------------------------------------------------------------------- the cases

def _pe(name, templates, T, fmax, lags, first, nodes, nb=200, nd=219, dtype="f32", loud=1024, random=1024,
        prior="volume", quadrature="reference", precision="reference", segments=1, snr=15.0, graph=False):
    return dict(name=name, kind="pe", templates=templates, T=T, fmax=fmax, lags=lags, first=first, nodes=nodes, nb=nb,
                nd=nd, dtype=dtype, loud=loud, random=random, prior=prior, quadrature=quadrature, precision=precision,
                segments=segments, snr=snr, graph=graph)


def listed():
    return [
        # a quick look at one segment with a small bank and a few nodes: launches and latency
        _pe("pe_64x3_8s_256Hz", 64, 8.0, 256.0, 43, 24, 3, nb=100, nd=109),
        # the small bank of the serving mix on short segments, every node, graph replay as the server runs it
        _pe("pe_256x53_4s_graph", 256, 4.0, 512.0, 87, 0, 53, graph=True),
        # the headline workload of the benchmark
        _pe("pe_2048x53_8s", 2048, 8.0, 512.0, 87, 0, 53),
        # long segments, tables kept in 16 bits
        _pe("pe_1024x53_16s_f16", 1024, 16.0, 512.0, 87, 0, 53, dtype="f16", snr=8.0),
        # the largest bank of the serving mix: its lags do not fit one pass
        _pe("pe_8192x53_4s", 8192, 4.0, 512.0, 87, 0, 53, snr=25.0),
        # ragged sizes, the float64 filter option, a tabulated prior with the Gauss-Legendre rule, two segments
        _pe("pe_333x21_6s_fp64", 333, 6.0, 400.0, 67, 27, 21, dtype="bf16", loud=700, random=451, prior="tabulated",
            quadrature="gl64", precision="fp64", segments=2, snr=30.0),
        # every arrival time walked (no selection), the tabulated prior
        _pe("pe_24x12_alltimes", 24, 4.0, 256.0, 43, 20, 12, loud=0, random=0, prior="tabulated"),
        # the published pe_redshift timing: 120 equal-mass templates on the default 1600 x 1600 grid
        dict(name="redshift_120_1600", kind="redshift", templates=120, T=8.0, fmax=512.0, lags=87, first=0, nodes=53,
             nb=200, nd=219, dtype="f32", nz=1600, nm1=1600, loud=1024, random=1024, snr=20.0),
        # the general gather contract at the reference's nodes_per_launch
        dict(name="gather_96x6", kind="gather", rows=96, slots=6, T=8.0, fmax=512.0, lags=87, first=24, nodes=6,
             nb=200, nd=219, walk=2048, snr=15.0),
        # the filter stage on its own, with the trajectories returned to the caller
        dict(name="trajectories_64_8s", kind="trajectories", templates=64, T=8.0, fmax=512.0, snr=15.0),
        # stage 1 at the published order for a few nodes (wtable's node indices) and pixels
        dict(name="wtable_n120_6nodes", kind="wtable", n_max=120, nodes=6, n_tau=5, pixels=3),
        # stages 2 and 3 of one node at the published order and grids, a share of its lags
        dict(name="tables_n120_12lags", kind="tables", n_max=120, lags=12, nq=110, nphi=96),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _lags(fmax):
    """lags of the H-L light travel time (10 ms, 5 % margin) at the filter's time step 1 / (8 fmax)"""
    return 2 * int(1.05 * 0.010013 * 8.0 * fmax) + 1


def draw(rng):
    kind = rng.choice(["pe"] * 6 + ["redshift", "gather", "trajectories", "wtable", "tables"])
    T, fmax = rng.choice([4.0, 6.0, 8.0, 12.0, 16.0]), rng.choice([256.0, 300.0, 400.0, 512.0])
    snr = round(rng.uniform(0.0, 40.0), 1)
    if kind == "pe":
        nodes = rng.choice([53, 53, rng.randint(3, 20)])
        first = 0 if nodes == 53 else rng.randint(24, 30)
        small = rng.random() < 0.2
        walk_all = rng.random() < 0.1
        c = _pe("", _log_int(rng, 24, 1600), T, fmax, _lags(fmax), first, nodes, nb=100 if small else 200,
                nd=109 if small else 219, dtype=rng.choice(["f32", "f32", "f16", "bf16"]),
                loud=0 if walk_all else _log_int(rng, 100, 1500), random=0 if walk_all else _log_int(rng, 100, 1500),
                prior=rng.choice(["volume", "volume", "tabulated"]), quadrature=rng.choice(["reference", "gl64"]),
                precision=rng.choice(["reference", "reference", "fp64"]), segments=rng.choice([1, 1, 2, 3]), snr=snr,
                graph=rng.random() < 0.3)
        if walk_all:
            c.update(templates=_log_int(rng, 8, 32), T=4.0)
        del c["name"]
        while _node_taps(c) > 1.2e10:
            c["templates"] = c["templates"] * 2 // 3
        return c
    if kind == "redshift":
        return dict(kind=kind, templates=rng.randint(40, 200), T=rng.choice([4.0, 8.0]), fmax=fmax, lags=_lags(fmax),
                    first=0, nodes=53, nb=200, nd=219, dtype="f32", nz=rng.randint(200, 1600),
                    nm1=rng.randint(200, 1600), loud=_log_int(rng, 200, 1024), random=_log_int(rng, 200, 1024), snr=snr)
    if kind == "gather":
        nodes = rng.randint(2, 6)
        return dict(kind=kind, rows=_log_int(rng, 8, 128), slots=rng.randint(1, nodes), T=rng.choice([4.0, 8.0]),
                    fmax=fmax, lags=_lags(fmax), first=rng.randint(20, 30), nodes=nodes, nb=200, nd=219,
                    walk=rng.choice([0, _log_int(rng, 200, 2048)]), snr=snr)
    if kind == "trajectories":
        return dict(kind=kind, templates=_log_int(rng, 8, 96), T=T, fmax=fmax, snr=snr)
    if kind == "wtable":
        n_max = _log_int(rng, 16, 96)
        return dict(kind=kind, n_max=n_max, nodes=rng.randint(1, 53 if n_max < 48 else 12), n_tau=rng.randint(3, 9),
                    pixels=_log_int(rng, 2, 24))
    return dict(kind="tables", n_max=_log_int(rng, 16, 120), lags=rng.randint(2, 12), nq=rng.randint(40, 110),
                nphi=rng.choice([32, 48, 64, 96]))


# ----------------------------------------------------------------------------- what a program keeps

_kept = {}


def _keep(key, make):
    if key not in _kept:
        _kept[key] = make()
    return _kept[key]


def _spec(c):
    return synth.TableSpec(ntau=c["lags"], nb=c["nb"], nd=c["nd"])


def _s_nodes(c):
    return synth.S_NODES_PROD[c["first"]:c["first"] + c["nodes"]]


def _make_store(c, dtype):
    spec, s = _spec(c), _s_nodes(c)
    store = synth.MemoryStore(spec, s, TABLE_SEED, tables=[None] * s.size, table_dtype=dtype)
    store.generator = (*spec.factors(s), TABLE_SEED)
    return store


def _store(c):
    dtype = c.get("dtype", "f32")
    return _keep(("store", c["lags"], c["nb"], c["nd"], c["first"], c["nodes"], dtype), lambda: _make_store(c, dtype))


def _segments(c, n, seed):
    return synth.make_segments(n, 1000 * (seed % (1 << 30)) + 7, T=c["T"], fmax=c["fmax"], snr=c["snr"],
                               mc=(15.0, 35.0), q=(0.4, 1.0), chi=(-0.3, 0.3))


def _rows(c):
    if c["kind"] == "redshift":
        M = np.geomspace(8.0, 150.0, c["templates"])
        return np.stack([M, np.ones_like(M), np.zeros_like(M)], axis=1)
    return synth.make_bank(c.get("templates", c.get("rows")), BANK_SEED)


def _bank(c):
    def make():
        seg = _segments(dict(c, snr=0.0), 1, 0)
        rows = _rows(c)
        return eb.MassBank(rows[:, 0], rows[:, 1], rows[:, 2], seg, "b200", profile=synth.profile)
    return _keep(("bank", c["kind"] == "redshift", _rows(c).shape[0], c["T"], c["fmax"]), make)


def _prior(c):
    """a smooth density of ln y, as a tabulated population prior gives it"""
    if c["prior"] == "volume":
        return "volume"
    lny = np.linspace(math.log(YMIN), math.log(60.0), 400)
    p = np.exp(-1.8 * (lny - lny[0])) * (1.0 - np.exp(-4.0 * (lny - lny[0]) - 0.2))
    return lny, p / np.trapezoid(p, lny)


def _rng_case(c, seed, salt):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, salt])


def _w_inputs(c, seed):
    """pixels spread over the nside-32 sky and the nodes of the published grid"""
    pix = np.sort(_rng_case(c, seed, 5).choice(wtable.nside2npix(wtable.NSIDE), c["pixels"], replace=False))
    return synth.S_NODES_PROD[np.linspace(4, 46, c["nodes"]).astype(int)], pix


def _table_inputs(c, seed):
    """one node's rebinned W over the keys (n, a, b <= a): decaying in a - b as the quadrature's moments do, with a
    per-key scatter and a lag profile; the magnitude grid"""
    rng = _rng_case(c, seed, 6)
    n_max, s = c["n_max"], 25.0
    keys = _keep(("keys", n_max), lambda: np.array(wtable.keys(n_max)))
    lnq = np.log(np.geomspace(0.05, 100.0, c["nq"]))
    base = np.exp(-0.8 * (keys[:, 1] - keys[:, 2]) - 0.05 * keys[:, 0])
    prof = np.exp(-0.5 * ((np.arange(c["lags"]) - c["lags"] / 2.0) / (1.0 + c["lags"] / 3.0)) ** 2)
    Wd = base[:, None] * prof[None, :] * (1.0 + 0.01 * rng.uniform(-1.0, 1.0, (keys.shape[0], c["lags"])))
    return keys, Wd, s, lnq


def prepare(case, seed):
    c = dict(case)
    if c["kind"] in ("pe", "redshift"):
        bank, store = _bank(c), _store(c)
        seg = _segments(c, c.get("segments", 1), seed)
        prior = _prior(c) if c["kind"] == "pe" else "volume"
        eb.prepare(bank, store, prior, YMIN, c.get("quadrature", "reference"))
        bank.ctx.set_graph(bool(c.get("graph", False)))
        return dict(case=c, bank=bank, store=store, seg=seg, prior=prior)
    if c["kind"] == "gather":
        store, bank = _make_store(c, "f32"), _bank(c)
        ctx = eb.Context(0)   # a context of the program's own: its trajectories and times stay resident
        own = bank.clone_for(ctx)
        eb.prepare(own, store, "volume", YMIN)
        traj, times = _traj_inputs(c, seed)
        ctx.set_trajectories({k: v for k, v in traj.items()})
        ctx.set_times(times)
        ids, lna, tab = _gather_slots(c, bank.u)
        return dict(case=c, ctx=ctx, store=store, ids=ids, lna=lna, tab=tab)
    if c["kind"] == "trajectories":
        small = dict(c, lags=43, nb=100, nd=109, first=20, nodes=8)
        bank = _bank(c)
        eb.prepare(bank, _store(small), "volume", YMIN)
        seg = eb.read_segments(_segments(c, 1, seed))
        return dict(case=c, bank=bank, d={I: seg["d_" + I][0] for I in "HL"}, sig2={I: seg["sig2_" + I] for I in "HL"})
    if c["kind"] == "wtable":
        s, pix = _w_inputs(c, seed)
        return dict(case=c, s=s, pix=pix, ctx=eb.context(0))
    keys, Wd, s, lnq = _table_inputs(c, seed)
    return dict(case=c, Wd=Wd, lnq=lnq, k=tables.k_inputs(keys, s, c["n_max"], lnq, c["nphi"]), ctx=eb.context(0))


def run(state):
    c = state["case"]
    if c["kind"] == "pe":
        r = eb.pe_intrinsic(state["seg"], state["bank"], state["store"], prior=state["prior"], ymin=YMIN,
                            n_loud=c["loud"], n_random=c["random"], seed=3, quadrature=c["quadrature"],
                            filter_precision=c["precision"])
        return dict(ln_lambda=r["ln_lambda"].astype(np.float32), ln_b=r["ln_b"].astype(np.float32))
    if c["kind"] == "redshift":
        r = eb.pe_redshift(state["seg"], state["bank"], state["store"], nz=c["nz"], nm1=c["nm1"], n_loud=c["loud"],
                           n_random=c["random"], seed=3)
        return dict(ln_lambda=torch.from_numpy(r["ln_lambda"]).float(), ln_b=r["ln_b"].astype(np.float32))
    if c["kind"] == "gather":
        return dict(out=state["ctx"].gather(state["ids"], state["lna"], state["tab"]))
    if c["kind"] == "trajectories":
        return state["bank"].trajectories(state["d"], state["sig2"])
    if c["kind"] == "wtable":
        return dict(W=wtable.w_table(state["s"], n_max=c["n_max"], n_tau=c["n_tau"], pixels=state["pix"],
                                     ctx=state["ctx"])[1])
    coeff, gmo, cosm = state["k"]
    col, row, _ = state["ctx"].k_edges(c["n_max"], state["Wd"], coeff, state["lnq"], gmo, cosm)
    return dict(T=tables.bd_tables(col, row, state["lnq"], ctx=state["ctx"])[0][c["n_max"]])


# ----------------------------------------------------------------------------- the work of a case

def _n_time(c):
    return 8 * int(c["fmax"] * c["T"])


def _n_freq(c):
    return int(c["fmax"] * c["T"]) - int(math.ceil(20.0 * c["T"])) + 1


def _node_taps(c):
    """(template, node slot, lag, walked time) table reads of a pe or redshift case: a template reaches about 45 of the 53
    nodes, and every node of a slice of the grid, plus its boundary point"""
    slots = 45.0 if c["nodes"] == 53 else c["nodes"]
    walk = (c["loud"] + c["random"]) if c["loud"] else _n_time(c)
    return c["templates"] * slots * c["lags"] * walk * c.get("segments", 1)


def work(case):
    c = case
    if c["kind"] in ("pe", "redshift"):
        nm, nt, nf, ns = c["templates"], _n_time(c), _n_freq(c), c.get("segments", 1)
        taps = _node_taps(c)
        # the part of the tables that the taps of a segment can reach: every lag and phase plane, about 80 rows of beta by
        # 160 of Delta, or 8 values per table read where that is less
        elem = 2 if c["dtype"] != "f32" else 4
        table = min(ns * c["nodes"] * c["lags"] * 49.0 * min(c["nb"], 80) * min(c["nd"], 160), 8.0 * taps) * elem
        out = 4.0 * ns * nm if c["kind"] == "pe" else 8.0 * c["nz"] * c["nm1"]
        data = nm * nf * 8.0 + ns * nf * 48.0 + out
        # 8-point interpolation and one exponential per table read; two transforms per template
        return {"bytes": table + data, "flops": 26.0 * taps + ns * 2.0 * nm * 5.0 * nt * math.log2(nt)}
    if c["kind"] == "gather":
        walk = c["walk"] or _n_time(c)
        taps = float(c["rows"]) * c["slots"] * c["lags"] * walk
        table = min(c["nodes"] * c["lags"] * 49.0 * 80 * 160, 8.0 * taps) * 4.0
        return {"bytes": table + c["rows"] * (walk * 16.0 + c["slots"] * 24.0), "flops": 40.0 * taps}
    if c["kind"] == "trajectories":
        nt, nm = _n_time(c), c["templates"]
        return {"bytes": 16.0 * nm * nt + 8.0 * nm * _n_freq(c), "flops": 2.0 * nm * 5.0 * nt * math.log2(nt)}
    n = c["n_max"]
    keys = (n + 1) * (n + 2) * (n + 3) / 6.0
    if c["kind"] == "wtable":
        q = (2 * n + 3) * (n + 3)
        return {"bytes": c["nodes"] * c["n_tau"] * keys * 4.0 + c["nodes"] * keys * 8.0,
                "flops": 2.0 * c["pixels"] * c["nodes"] * q * keys}
    nqb, nphif = 2 * c["nq"] - 1, c["nphi"] // 2 + 1
    nb = tables.bd_grid(np.log(np.geomspace(0.05, 100.0, c["nq"])))[0].size
    out = float(c["lags"]) * nphif * nb * nqb
    return {"bytes": keys * c["lags"] * 8.0 + out * 4.0,
            "flops": 2.0 * keys * c["lags"] * nqb + (n + 1) * (n + 2.0) * c["lags"] * nqb * nphif + 8.0 * out * (n + 1)}


# ----------------------------------------------------------------------------- the same in 64 bits

def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _filter64(W, d, sig2, lo, nt):
    """ln|z| and arg z of the matched filter, complex128"""
    w = torch.from_numpy(np.conj(d) / sig2).to(_dev())
    lq, ph = [], []
    for i in range(0, W.shape[0], 512):
        pad = torch.zeros((min(512, W.shape[0] - i), nt), dtype=torch.complex128, device=_dev())
        pad[:, lo:lo + W.shape[1]] = torch.from_numpy(W[i:i + 512]).to(_dev()).to(torch.complex128) * w[None, :]
        z = torch.fft.fft(pad, dim=-1)
        lq.append(0.5 * torch.log(torch.clamp(z.real ** 2 + z.imag ** 2, min=1e-38)))
        ph.append(torch.atan2(z.imag, z.real))
    return torch.cat(lq), torch.cat(ph)


def _select(lqH, lqL, lags, K, S, seed):
    """the n_loud loudest times by the float32 score, n_random numpy draws from the rest, sorted: (times, random?)"""
    nm, nt = lqH.shape
    if K == 0:
        return torch.arange(nt, device=_dev()).expand(nm, nt), torch.zeros((nm, nt), dtype=torch.bool, device=_dev())
    h = lags // 2
    H = lqH.float()
    mx = torch.nn.functional.max_pool1d(torch.cat([H[:, nt - h:], H, H[:, :h]], dim=1)[None], 2 * h + 1, 1)[0]
    score = np.exp(2 * lqL.float().cpu().numpy()) + np.exp(2 * mx.cpu().numpy())
    top = torch.topk(torch.from_numpy(score).to(_dev()), K, dim=1).indices
    taken = torch.zeros((nm, nt), dtype=torch.int8, device=_dev()).scatter_(1, top, 1)
    rest = torch.argsort(taken, dim=1, stable=True)[:, :nt - K]
    pick = torch.from_numpy(np.random.default_rng(seed).integers(0, nt - K, size=(nm, S))).to(_dev())
    t, order = torch.sort(torch.cat([top, torch.gather(rest, 1, pick)], dim=1), dim=1)
    return t, order >= K


def _mix32(h):
    m = 0xFFFFFFFF
    h = h ^ (h >> 16)
    h = (h * 0x7FEB352D) & m
    h = h ^ (h >> 15)
    h = (h * 0x846CA68B) & m
    return h ^ (h >> 16)


def _table(spec, fac, k, r):
    """the store's float32 table of node k at lag row r, (49, nb, nd)"""
    M, P, Q, S = fac
    m = 0xFFFFFFFF
    ar = lambda n: torch.arange(n, dtype=torch.int64, device=_dev())  # noqa: E731
    h = torch.tensor(((TABLE_SEED * 0x9E3779B1) & m) ^ ((k * 0x85EBCA77) & m), dtype=torch.int64, device=_dev())
    h = _mix32(h ^ ((r * 0xC2B2AE3D) & m))
    h = _mix32(h ^ ((ar(spec.nphif) * 0x27D4EB2F) & m))
    h = _mix32(h[:, None] ^ ((ar(spec.nb) * 0x165667B1) & m)[None, :])
    h = _mix32(h[:, :, None] ^ ((ar(spec.nd) * 0xD3A2646C) & m)[None, None, :])
    v = torch.from_numpy(M).to(_dev())[None] * torch.from_numpy(P).to(_dev())[:, None, None]
    v = v * float(Q[r])
    v = v - float(S[k])
    return v + ((h & 0xFFFF) - 32768).float() * 2.0 ** -22


def _stored(T, dtype, node_max):
    """the values a 16-bit store holds for float32 table values"""
    if dtype == "bf16":
        return T.bfloat16().float()
    if dtype == "f16":
        scale = 2.0 ** (math.frexp(node_max)[1] - 15)
        return (T * (1.0 / scale)).half().float() * scale
    return T


def _read64(lqH, phH, lqL, phL, t, random, lw, spec, fac, slots, dtype="f32", phase32=False):
    """Eq. (C7) in float64: slots is a list of (node, template rows, ln a); returns for each the (rows,) log-sum-exp over
    lags and visited times minus ln n_time"""
    nt = lqH.shape[1]
    b0, db, d0, dd = (float(spec.beta[0]), float(spec.beta[1] - spec.beta[0]), float(spec.delta[0]),
                      float(spec.delta[1] - spec.delta[0]))
    nb, nd, nphif = spec.nb, spec.nd, spec.nphif
    add = torch.where(random, lw, 0.0)
    aL, pL = torch.gather(lqL, 1, t), torch.gather(phL, 1, t)
    acc = [[] for _ in slots]
    top = {}
    if dtype == "f16":
        for k in {s[0] for s in slots}:
            top[k] = max(float(_table(spec, fac, k, r).abs().max()) for r in range(spec.ntau))
    for r, tau in enumerate(spec.tau_idx):
        i1 = (t + int(tau)) % nt
        aH, pH = torch.gather(lqH, 1, i1), torch.gather(phH, 1, i1)
        dph = (pH.float() - pL.float()).double() if phase32 else pH - pL
        x3 = dph * (NPHI / (2.0 * math.pi))
        x3 = torch.where(x3 < 0, x3 + NPHI, x3)
        x3 = torch.where(x3 >= NPHI, x3 - NPHI, x3)
        c0 = x3.long().clamp(0, NPHI - 1)
        fc = x3 - c0
        c1 = (c0 + 1) % NPHI
        c0, c1 = (torch.where(c > NPHI // 2, NPHI - c, c) * (nb * nd) for c in (c0, c1))
        have = None
        for j, (k, rows, lna) in enumerate(slots):
            if have != k:
                tab, have = _stored(_table(spec, fac, k, r), dtype, top.get(k, 1.0)).double().reshape(-1), k
            every = rows.numel() == t.shape[0]
            part = (lambda v: v) if every else (lambda v: v[rows])
            l = part(aL)
            xr = l * (2.0 / db) + ((lna - b0) / db)[:, None]
            xb = xr.clamp(0.0, nb - 1 - 1e-6)
            xd = ((part(aH) - (l + (xb - xr) * (db / 2.0))) / dd - d0 / dd).clamp(0.0, nd - 1 - 1e-6)
            ib, id_ = xb.long(), xd.long()
            fb, fd = xb - ib, xd - id_
            at, w = ib * nd + id_, part(fc)
            v = 0.0
            for c, wc in ((part(c0), 1.0 - w), (part(c1), w)):
                o = c + at
                v = v + wc * ((1 - fb) * ((1 - fd) * tab[o] + fd * tab[o + 1])
                              + fb * ((1 - fd) * tab[o + nd] + fd * tab[o + nd + 1]))
            acc[j].append(torch.logsumexp(v + part(add), dim=1))
    return [torch.logsumexp(torch.stack(a), dim=0) - math.log(nt) for a in acc]


def _geometry(spec_s, u):
    """valid (node, template) pairs, y of every point and the boundary point's node and ln a"""
    alo, ahi = min(float(synth.ALPHA[0]), YMIN * YMIN), float(synth.ALPHA[-1])
    a = spec_s[:, None] / u[None, :]
    valid = (np.sqrt(a) >= YMIN) & (a > alo) & (a < ahi)
    before = np.concatenate([[0.0], spec_s[:-1]])[:, None] / u[None, :]
    low = valid & (before <= alo)
    bnode = np.where(low.any(0), low.shape[0] - 1 - np.argmax(low[::-1], axis=0), -1)
    a_b = alo * (1.0 + 1e-9)
    y = np.where(valid, np.sqrt(a), 0.0)
    return valid, np.log(a), np.concatenate([y, np.where(bnode >= 0, math.sqrt(a_b), 0.0)[None]]), bnode, math.log(a_b)


def _node_values64(c, bank, spec, fac, d, sig2, seed):
    lq, ph = {}, {}
    for I in "HL":
        lq[I], ph[I] = _filter64(bank.W, d[I], sig2[I], bank.lo, bank.n_time)
    t, rnd = _select(lq["H"], lq["L"], spec.ntau, c["loud"], c["random"], seed)
    lw = math.log((bank.n_time - c["loud"]) / c["random"]) if c["loud"] else 0.0
    valid, lna, y, bnode, lna_b = _geometry(_s_nodes(c), np.asarray(bank.u))
    nn, nm = valid.shape
    slots = []
    for k in range(nn):
        for rows, la in ((np.nonzero(valid[k])[0], lna[k]), (np.nonzero(bnode == k)[0], np.full(nm, lna_b))):
            if rows.size:
                slots.append((k, torch.from_numpy(rows).to(_dev()), torch.from_numpy(la[rows]).to(_dev())))
    got = _read64(lq["H"], ph["H"], lq["L"], ph["L"], t, rnd, lw, spec, fac, slots, c["dtype"])
    lam = np.full((nn + 1, nm), -np.inf)
    seen = set()
    for (k, rows, _), v in zip(slots, got):
        bound = k in seen or not valid[k].any()
        seen.add(k)
        lam[nn if bound else k, rows.cpu().numpy()] = v.cpu().numpy()
    return lam, y


def _ln_weights(y, prior, gl):
    """ln of the weights that integrate the distance prior against a function linear in ln y between a template's points"""
    out = np.full(y.shape, -np.inf)
    gx, gw = np.polynomial.legendre.leggauss(64)
    for m in range(y.shape[1]):
        pts = np.nonzero(y[:, m] > 0)[0]
        pts = pts[np.argsort(y[pts, m])]
        x = np.log(y[pts, m])
        a, b = x[:-1, None], x[1:, None]
        h = (b - a)[:, 0]
        if gl:
            t = 0.5 * (a + b) + 0.5 * (b - a) * gx
        else:
            t = a + (b - a) * np.linspace(0.0, 1.0, 401)
        f = 3.0 * YMIN ** 3 * np.exp(-3.0 * t) if isinstance(prior, str) else np.interp(t, *prior, left=0.0, right=0.0)
        if gl:
            lo, hi = (0.5 * np.sum(gw * f * g, axis=1) for g in (b - t, t - a))
        elif isinstance(prior, str):
            a, b = a[:, 0], b[:, 0]
            ea, eb_ = np.exp(-3.0 * a), np.exp(-3.0 * b)
            i0 = (ea - eb_) / 3.0
            i1 = (a * ea - b * eb_) / 3.0 + (ea - eb_) / 9.0
            lo, hi = (3.0 * YMIN ** 3 * v / h for v in (b * i0 - i1, i1 - a * i0))
        else:
            lo, hi = (np.trapezoid(f * g / h[:, None], t, axis=1) for g in (b - t, t - a))
        w = np.zeros(pts.size)
        w[:-1] += lo
        w[1:] += hi
        with np.errstate(divide="ignore"):
            out[pts, m] = np.log(w)
    return out


def _log_mean(lam, w):
    ok = np.isfinite(lam) & (w > 0)
    top = lam[ok].max()
    return top + math.log(float(np.sum(w[ok] * np.exp(lam[ok] - top))))


def _cells(bank):
    cell = np.ones(bank.M.size)
    for ax in (bank.M, bank.q, bank.chi):
        vals = np.unique(ax)
        if vals.size > 1:
            cell *= np.gradient(vals)[np.searchsorted(vals, ax)]
    return cell / cell.sum()


def _exact_pe(c, seed):
    bank, spec = _bank(c), _spec(c)
    fac, seg = spec.factors(_s_nodes(c)), _segments(c, c["segments"], seed)
    L, lnw = [], None
    for e in range(c["segments"]):
        lam, y = _node_values64(c, bank, spec, fac, {I: seg["d_" + I][e] for I in "HL"},
                                {I: seg["sig2"] for I in "HL"}, 3 + e)
        lnw = _ln_weights(y, _prior(c), c["quadrature"] == "gl64") if lnw is None else lnw
        L.append(np.logaddexp.reduce(lnw + lam, axis=0))
    cell = _cells(bank)
    return dict(ln_lambda=np.array(L), ln_b=np.array([_log_mean(v, cell) for v in L]))


def _exact_redshift(c, seed):
    bank, spec = _bank(c), _spec(c)
    fac, seg = spec.factors(_s_nodes(c)), _segments(c, 1, seed)
    lam, y = _node_values64(c, bank, spec, fac, {I: seg["d_" + I][0] for I in "HL"}, {I: seg["sig2"] for I in "HL"}, 3)
    from exmarg_b200.cosmology import dl_of_z   # the distances are an input of the analysis
    z, m1 = np.linspace(0.02, 8.0, c["nz"]), np.geomspace(3.0, 150.0, c["nm1"])
    dl = _keep(("dl", c["nz"]), lambda: dl_of_z(z))
    yq, M = D0 / dl, np.asarray(bank.M)
    surf = np.full((c["nz"], M.size), -np.inf)
    for m in range(M.size):
        ok = np.isfinite(lam[:, m]) & (y[:, m] > 0)
        if ok.sum() >= 2:
            o = np.argsort(y[ok, m])
            surf[:, m] = np.interp(yq, y[ok, m][o], lam[ok, m][o], left=-np.inf, right=-np.inf)
    out = np.full((c["nm1"], c["nz"]), -np.inf)
    for i in range(c["nz"]):
        ok = np.isfinite(surf[i])
        if ok.sum() >= 2:
            out[:, i] = np.interp(2.0 * m1 * (1.0 + z[i]), M[ok], surf[i, ok], left=-np.inf, right=-np.inf)
    Md = 2.0 * m1[:, None] * (1.0 + z[None, :])
    w = np.where((Md >= 10.0) & (Md <= 500.0), np.exp(np.log(np.maximum((1 + z) * dl ** 2 * np.gradient(dl, z), 1e-300)))[None, :],
                 0.0) * np.gradient(m1)[:, None] * np.gradient(z)[None, :]
    return dict(ln_lambda=out[None], ln_b=np.array([_log_mean(out, w / w.sum())]))


def _traj_inputs(c, seed):
    """float32 trajectories of one segment and the visited times with their log weights (None: every time), host arrays"""
    bank = _bank(c)
    seg = _segments(c, 1, seed)
    traj = {}
    for I in "HL":
        lq, ph = _filter64(bank.W, seg["d_" + I][0], seg["sig2"], bank.lo, bank.n_time)
        traj["lq" + I], traj["ph" + I] = lq.float().cpu().numpy(), ph.float().cpu().numpy()
    if not c["walk"]:
        return traj, None
    K = c["walk"] // 2
    S = c["walk"] - K
    t, rnd = _select(torch.from_numpy(traj["lqH"]).to(_dev()), torch.from_numpy(traj["lqL"]).to(_dev()), c["lags"], K, S, 3)
    lw = np.float32(math.log((bank.n_time - K) / S))
    return traj, (t.cpu().numpy().astype(np.int32), np.where(rnd.cpu().numpy(), lw, np.float32(0.0)))


def _gather_slots(c, u):
    """each row reads `slots` consecutive nodes, rotated from row to row"""
    ids = np.arange(c["rows"])
    tab = (ids[:, None] + np.arange(c["slots"])[None, :]) % c["nodes"]
    return ids, np.log(_s_nodes(c)[tab] / np.asarray(u)[:, None]), tab


def _exact_gather(c, seed):
    spec, bank = _spec(c), _bank(c)
    traj, times = _traj_inputs(c, seed)
    tr = {k: torch.from_numpy(v).to(_dev()).double() for k, v in traj.items()}
    nt = bank.n_time
    if times is None:
        t = torch.arange(nt, device=_dev()).expand(c["rows"], nt)
        rnd, lw = torch.zeros(t.shape, dtype=torch.bool, device=_dev()), 0.0
    else:
        t, rnd, lw = torch.from_numpy(times[0]).long().to(_dev()), torch.from_numpy(times[1] != 0).to(_dev()), float(times[1].max())
    ids, lna, tab = _gather_slots(c, bank.u)
    slots, where = [], []
    for k in range(c["nodes"]):
        for n in range(c["slots"]):
            rows = np.nonzero(tab[:, n] == k)[0]
            if rows.size:
                slots.append((k, torch.from_numpy(rows).to(_dev()), torch.from_numpy(lna[rows, n]).to(_dev())))
                where.append((n, rows))
    out = np.empty((c["slots"], c["rows"]))
    for (n, rows), v in zip(where, _read64(tr["lqH"], tr["phH"], tr["lqL"], tr["phL"], t, rnd, lw, spec,
                                           spec.factors(_s_nodes(c)), slots, phase32=True)):
        out[n, rows] = v.cpu().numpy()
    return dict(out=out)


def _exact_wtable(c, seed):
    s, pix = _w_inputs(c, seed)
    n_max = c["n_max"]
    g = wtable.geometry(wtable.NSIDE, n_max, c["n_tau"], pix)   # antenna responses, delays and quadrature: inputs
    to = lambda v: torch.from_numpy(np.asarray(v, np.float64)).to(_dev())  # noqa: E731
    c2p, s2p, ap, cg, sj = to(g["c2p"]), to(g["s2p"]), to(g["ap"]), to(g["cg"]), to(s)
    wq = to(g["wq"])[None, :].expand(c2p.numel(), -1).reshape(-1)
    nk = (n_max + 1) * (n_max + 2) * (n_max + 3) // 6
    W = torch.zeros((len(s), c["n_tau"], nk), dtype=torch.float64, device=_dev())
    for p in range(len(pix)):
        R = []
        for i in range(2):
            fp, fx = float(g["resp"][p, 2 * i]), float(g["resp"][p, 2 * i + 1])
            R.append(torch.complex((fp * c2p - fx * s2p)[:, None] * ap, (fp * s2p + fx * c2p)[:, None] * cg).reshape(-1))
        q1, q2 = (r.abs() / math.sqrt(2.0) for r in R)
        dph = R[0].angle() - R[1].angle()
        bw = torch.exp(-2.0 * sj[:, None] * (q1 ** 2 + q2 ** 2)) * wq
        e = torch.arange(n_max + 1, device=_dev())
        for m in range(n_max + 1):
            x, y = torch.meshgrid(e[:n_max - m + 1], e[:n_max - m + 1], indexing="ij")
            x, y = (v[x + y <= n_max - m] for v in (x, y))
            n, a, b = m + x + y, m + x, x
            A = bw * torch.cos(m * dph)
            P1 = q1[:, None] ** (m + 2 * e[:n_max - m + 1]).double()
            P2 = q2[:, None] ** (m + 2 * e[:n_max - m + 1]).double()
            key = n * (n + 1) * (n + 2) // 6 + a * (a + 1) // 2 + b
            for i in range(0, key.numel(), 2048):
                v = A @ (P1[:, x[i:i + 2048]] * P2[:, y[i:i + 2048]])
                for j in range(2):
                    W[:, int(g["j0"][p]) + j, key[i:i + 2048]] += float(g["w"][p, j]) * v
    order = np.repeat(np.arange(n_max + 1), [(k + 1) * (k + 2) // 2 for k in range(n_max + 1)])
    ln = order[None] * np.log(2.0 * s)[:, None] - np.array([math.lgamma(k + 1.0) for k in range(n_max + 1)])[order][None]
    return dict(W=(W * to(np.exp(np.minimum(ln, 700.0)))[:, None, :]).cpu().numpy())


def _exact_tables(c, seed):
    keys, Wd, s, lnq = _table_inputs(c, seed)
    n_max, nq, nphif = c["n_max"], c["nq"], c["nphi"] // 2 + 1
    to = lambda v: torch.from_numpy(np.asarray(v, np.float64)).to(_dev())  # noqa: E731
    W, l = to(Wd), to(lnq)
    last = float(lnq[-1])
    # Delta ascending: (q1, q_last) for q1 = 0 .. last, then (q_last, q2) for q2 = last - 1 .. 0
    l1 = torch.cat([l, torch.full((nq - 1,), last, dtype=torch.float64, device=_dev())])
    l2 = torch.cat([torch.full((nq,), last, dtype=torch.float64, device=_dev()), l.flip(0)[1:]])
    phi = torch.arange(nphif, dtype=torch.float64, device=_dev()) * (2.0 * math.pi / c["nphi"])
    beta = to(tables.bd_grid(lnq)[0])
    g = torch.empty((n_max + 1, c["lags"], nphif, 2 * nq - 1), dtype=torch.float64, device=_dev())
    for n in range(n_max + 1):
        base = n * (n + 1) * (n + 2) // 6
        C = []
        for m in range(n + 1):
            a = np.arange(m, n + 1)
            b = a - m
            co = np.array([math.comb(n, int(i)) * math.comb(n, int(j)) for i, j in zip(a, b)], float) * (2.0 if m else 1.0)
            e = to(a + b)[:, None]
            # relative to 2n max(l1, l2) = 2n last; g_n takes 2n l2 off again
            P = torch.exp(e * l1 + (2 * n - e) * l2 - 2 * n * last)
            C.append((to(co)[:, None] * W[torch.from_numpy(base + a * (a + 1) // 2 + b).to(_dev())]).T @ P)
        K = torch.einsum("mtq,mp->tpq", torch.stack(C), torch.cos(torch.arange(n + 1, device=_dev())[:, None] * phi))
        g[n] = torch.log(K) + 2 * n * last - (math.lgamma(n + 1.0) + n * math.log(s)) - 2 * n * l2
    out = np.empty((c["lags"], nphif, beta.numel(), 2 * nq - 1))
    nbeta = torch.arange(n_max + 1, device=_dev())[:, None] * beta
    for t in range(c["lags"]):
        for p in range(nphif):
            out[t, p] = torch.logsumexp(nbeta[:, :, None] + g[:, t, p][:, None, :], dim=0).cpu().numpy()
    return dict(T=out)


def exact(case, seed):
    c = dict(case)
    if c["kind"] in ("pe", "redshift") and _node_taps(c) > 2e10:
        return None   # over 20 seconds in 64 bits
    if c["kind"] == "trajectories":
        bank, seg, out = _bank(c), _segments(c, 1, seed), {}
        for I in "HL":
            lq, ph = _filter64(bank.W, seg["d_" + I][0], seg["sig2"], bank.lo, bank.n_time)
            out["lq" + I], out["ph" + I] = lq.cpu().numpy(), ph.cpu().numpy()
        return out
    return {"pe": _exact_pe, "redshift": _exact_redshift, "gather": _exact_gather, "wtable": _exact_wtable,
            "tables": _exact_tables}[c["kind"]](c, seed)
