"""Large copies between pageable host arrays and the device (csrc/hostio.cu) in both directions, at sizes on either
side of the plain copy's limit (2 MiB) and of the slots (1 MiB): trajectories read back and uploaded again give bitwise the
node values of the trajectories that never left the device, and the read-back ones are the float64 filter's to float32
rounding."""

import numpy as np
import pytest

import exmarg_b200 as eb
from exmarg_b200 import synth
from oracle import restate

pytestmark = pytest.mark.gpu


# four float32 planes of nm x 8 nu_max: 1.9, 2.0, 2.1, 5.6 and 12.6 MB
@pytest.mark.parametrize("nm, nu_max", [(29, 512), (32, 512), (33, 512), (43, 1021), (77, 1280)])
def test_trajectories_there_and_back(nm, nu_max):
    T, fmax = 4.0, nu_max / 4.0
    spec = synth.TableSpec(ntau=9, nb=100, nd=109)
    store = synth.MemoryStore(spec, synth.S_NODES_PROD[26:29], 5)
    seg = synth.make_segments(1, 40 + nm, T=T, fmax=fmax, snr=12.0, mc=10.0)
    rows = synth.make_bank(nm, 9, mc=(8.0, 15.0))
    ctx = eb.Context(0)
    try:
        bank = eb.MassBank(rows[:, 0], rows[:, 1], rows[:, 2], seg, profile=synth.profile).clone_for(ctx)
        eb.prepare(bank, store, "volume", 0.1267)
        assert bank.n_time == 8 * nu_max
        sg = eb.read_segments(seg)
        traj = bank.trajectories({I: sg["d_" + I][0] for I in "HL"}, {I: sg["sig2_" + I] for I in "HL"})
        here = ctx.node_values(3)
        ctx.set_trajectories(traj)
        back = ctx.node_values(3)
    finally:
        ctx.close()
    assert np.array_equal(here, back)
    want = restate.trajectories(bank.W, {I: sg["d_" + I][0] for I in "HL"}, {I: sg["sig2_" + I] for I in "HL"}, bank.lo,
                                bank.n_time)
    for I in "HL":
        # complex64 products: a few 2^-24 of the filter's largest value, relative to |z| at the sample
        rel = 8 * 2.0 ** -24 * np.exp(want["lq" + I].max(axis=1, keepdims=True) - want["lq" + I]) + 2.0 ** -20
        assert (np.abs(traj["lq" + I] - want["lq" + I]) <= rel).all()
