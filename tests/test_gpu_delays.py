"""Stepping in windows of the shortest delay, at the edges of its rings: delays of one
step, below, at and above the longest window, multiples of each other and not, sizes
around a warp and a tile, launches that split windows, and background rates on both sides
of the window-wide draw's limits.  Rasters and activity must equal the FP64 oracle's, and
every state of both forms must equal, bit for bit, what one launch per step gave (digests
in golden/delay_states.json; the oracle's states are no such measure here: the last bit of
its exp grows to 1e-10 in an upstroke)."""
import hashlib
import json
from pathlib import Path

import numpy as np
import pytest

import astrosimgpu_cuda_b200 as asg
from oracle import oracle

pytestmark = pytest.mark.gpu

STATE = ("V", "w", "g_ex", "dg_ex", "g_in", "dg_in", "I_sic", "stp_x", "stp_u", "stp_t_last",
         "Ca", "IP3", "h", "sic_factor")
GOLDEN = Path(__file__).parent / "golden" / "delay_states.json"

BUSY = {"w_e": 25.0, "SIC_th": 0.0715, "w_a2n": 3.0, "sic_interval": 2}

CASES = {}
for _d in ((0.1, 0.1, 0.1), (0.1, 0.3, 2.0), (0.4, 0.8, 1.2), (0.7, 1.1, 0.5), (1.6, 1.7, 1.6), (1.7, 1.7, 1.7),
           (2.0, 4.1, 3.3)):
    CASES["delays %g %g %g" % _d] = (dict(BUSY, d_e=_d[0], d_i=_d[1], d_a2n=_d[2]), (1, 4, 16, 29, 50),
                                     dict(n_total=700, seed=6))
for _n in (1, 2, 41, 161, 1281):
    for _b in (0, 32, 96, 640):
        CASES[f"size {_n} block {_b}"] = (dict(BUSY, d_e=0.6, d_i=1.6, d_a2n=1.0), (3, 47, 50),
                                          dict(n_total=_n, seed=_n, block=_b))
for _r in (0.0, 39990.0, 40010.0, 150000.0, 310000.0):
    CASES[f"rate {_r:g}"] = ({"d_i": 0.5, "exc_poiss_rate": _r, "inh_poiss_rate": 2500.0, "exc_poiss_weight": 0.02},
                             (3, 97), dict(n_total=300, seed=3))


def run(case, precision):
    """The stepped simulation and the digest of its states and raster."""
    bio, chunks, kw = CASES[case]
    sim = asg.Simulation(biology=bio, precision=precision, pre_ms=3.0, sim_ms=17.0, raster_steps=200, **kw)
    for c in chunks:
        sim.step(c)
    h = hashlib.sha256()
    for name in STATE:
        h.update(np.ascontiguousarray(sim.state(name)).tobytes())
    h.update(sim.raster().tobytes())
    return sim, h.hexdigest()[:16]


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("case", CASES)
def test_states(case, precision):
    sim, digest = run(case, precision)
    with sim:
        if precision == "fp64":
            bio, chunks, kw = CASES[case]
            o = oracle.OracleSim(biology=bio, pre_ms=3.0, sim_ms=17.0, raster_steps=200, **kw)
            o.step(sum(chunks))
            np.testing.assert_array_equal(sim.raster(), o.raster())
            a, b = sim.summary(), o.summary()
            for k in ("spikes_total", "active_astro", "engaged_astro"):
                assert a[k] == b[k], k
    assert digest == json.loads(GOLDEN.read_text())[case][precision]
