"""Stage 1's row tiles: exm_w_build takes 1, 2, 4 or 8 groups of the fewest rows that hold the nodes (1 to 8 rows each, the
threads left over sharing out the quadrature points), at the sizes on either side of each limit, with orders whose
quadrature does not fill its last step.  Against the float64 oracle, with the bar of the other stage-1 tests: 1e-7 of the
largest |W| of each (node, key), beyond two float32 subnormal steps (float64 sums in another order, one float32 rounding)."""

import numpy as np
import pytest

from exmarg_b200 import wtable
from oracle import restate

pytestmark = pytest.mark.gpu


def check(nodes, n_max):
    s = np.geomspace(0.05, 300.0, nodes) if nodes > 1 else np.array([3.0])
    _, W, _ = wtable.w_table(s, n_max, 1, 7)
    _, ref = restate.w_table_s(s, n_max, 1, 7, wtable.pix2ang, "correct")
    scale = np.abs(ref).max(axis=1, keepdims=True)
    err = np.maximum(np.abs(W.astype(np.float64) - ref) - 2.0 ** -148, 0.0) / np.maximum(scale, 1e-300)
    assert W.shape == ref.shape and float(err.max()) < 1e-7


@pytest.mark.parametrize("nodes, n_max", [(1, 0), (1, 9), (8, 9), (9, 17), (16, 5), (17, 9), (32, 5), (33, 9)])
def test_row_tiles_match_the_oracle(nodes, n_max):
    check(nodes, n_max)


@pytest.mark.parametrize("nodes", [2, 3, 4, 5, 6, 7, 10, 12, 14, 20, 21, 28, 40, 48, 49, 56, 64])
def test_every_row_count_matches_the_oracle(nodes):
    check(nodes, 6)
