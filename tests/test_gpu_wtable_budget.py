"""exm_w_build within the device memory of its inputs, ladders, sums and result: the cosines of a pixel take no memory of
their own beside a result that is as large."""

import numpy as np
import pytest

import exmarg_b200 as eb
from exmarg_b200 import wtable

pytestmark = pytest.mark.gpu


def test_the_cosines_share_the_results_memory():
    s, n_max, n_tau = np.geomspace(0.05, 300.0, 12), 24, 33
    pixels = np.arange(2)
    g = wtable.geometry(1, n_max, n_tau, pixels)
    keys, Q = (n_max + 1) * (n_max + 2) * (n_max + 3) // 6, g["c2p"].size * g["ap"].size
    assert s.size * n_tau * keys * 4 >= (n_max + 1) * Q * 8
    Qp = -(-Q // 32) * 32                                       # points of whole steps
    need = s.size * n_tau * keys * (8 + 4)                      # sums and result
    need += 2 * (2 * n_max + 1) * Qp * 8 + (1 + s.size) * Qp * 8    # ladders, phases, dampings
    need += s.size * (keys + 1) * 8 + pixels.size * 16 + g["c2p"].size * 8 + g["ap"].size * 16   # inputs
    tiles = sum(-(-(n + 1) // 8) * -(-(n + 1) // 16) for n in range(n_max + 1))
    need += tiles * 16 + 16 * 256                               # and the least allocations
    _, want, _ = wtable.w_table(s, n_max, 1, n_tau, pixels)
    ctx = eb.Context(0, hbm_budget=need)
    try:
        _, got, _ = wtable.w_table(s, n_max, 1, n_tau, pixels, ctx=ctx)
    finally:
        ctx.close()
    assert np.array_equal(got, want)
