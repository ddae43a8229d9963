"""The serving estimate of a worker's device memory against the arrays that a worker allocates, on the CPU."""

import pytest

from exmarg_b200.serve import workspace_bytes


@pytest.mark.parametrize("nm, n_time, nodes, lags, nfreq, walk", [
    (2048, 32768, 53, 87, 3937, 2048),    # the filter's rows and the descriptors share memory
    (2048, 2048, 53, 87, 240, 200),       # short segments, few times: the padding of the descriptors' runs counts
    (512, 4096, 12, 87, 500, 64),
    (8192, 8192, 53, 87, 1000, 2048),     # lags in several passes
])
def test_estimate_is_what_a_worker_allocates(nm, n_time, nodes, lags, nfreq, walk):
    per_pass = min(lags, (8 << 30) // (20 * nm * walk))
    taps = nm * walk + 3 * nm * min(48, walk)                 # of a lag, its (pair, template) runs in groups of four
    arrays = max(32 * nm * n_time, 16 * per_pass * taps)      # the filter's rows, then the descriptors
    arrays += 4 * per_pass * taps                             # time indices
    arrays += (16 + 8 + 4) * nm * n_time                      # trajectories, their residuals, scores
    arrays += 4 * per_pass * 48 * (nm + 1)                    # offsets of the runs
    arrays += 8 * (nodes + 1) * nm * (lags + 2)               # partial sums, node values, distance weights
    arrays += 8 * nm * nfreq + 4 * nm * walk                  # bank, visited times
    arrays += 32 * nm * n_time                                # cuFFT's work area
    est = workspace_bytes(nm, n_time, nodes, lags, nfreq, walk)
    assert arrays <= est <= 1.1 * arrays + (80 << 20)
