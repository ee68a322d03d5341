"""The parallel connectivity builder against the oracle's sequential walk, entry by entry:
sizes whose sections run with chunks of 2048, 4096, 8192 and 16384 tape positions, with
seeds that the stored digests do not cover."""
import numpy as np
import pytest

import astrosimgpu_cuda_b200 as asg
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_total,seed", [(2000, 5), (17011, 11), (30011, 12), (70001, 13), (150001, 14),
                                          (300000, 1), (300000, 2), (300000, 3)])
def test_every_entry(n_total, seed, monkeypatch):
    monkeypatch.setenv("ASTROSIM_BUILDER", "parallel")
    o = oracle.OracleSim(n_total=n_total, seed=seed, pre_ms=0, sim_ms=0)
    with asg.Simulation(n_total=n_total, seed=seed, pre_ms=0, sim_ms=0) as sim:
        for k in ("exc", "inh", "sic", "e2a"):
            (rs, src), (ors, osrc) = sim.csr(k), o.csr(k)
            assert osrc.size > 0
            np.testing.assert_array_equal(rs, ors, err_msg=k)
            np.testing.assert_array_equal(src, osrc, err_msg=k)
