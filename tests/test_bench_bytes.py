"""bench.py's byte model of a window against the DRAM traffic that ncu counted for one (no
GPU): what must move is no more than what moved, and most of it, at the profiled size, whose
state is several times the L2."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_the_model_fits_the_profiled_window(precision):
    prof = bench.PROFILED_WINDOW[precision]
    n = prof["n"]
    # the network's sizes follow from n; about 67 spikes a step and no active astrocyte when captured
    sizes = {"n_exc": int(0.8 * n), "n_inh": int(0.2 * n), "n_astro": int(0.2 * n), "n_exc_edges": 80 * n,
             "n_inh_edges": 20 * n, "n_e2a_edges": 16 * n, "n_sic_edges": 16 * n, "active_astro": 0}
    window = 10 * bench.window_step_bytes(sizes, precision, spikes_per_step=67.0)
    assert 0.9 * prof["dram"] < window <= prof["dram"]
