"""The windowed engine against one launch per step: digests of every state, spike count and
raster bit that an engine which draws, gathers and rounds every step by itself gave for the
same runs (golden/window_states.json).  Tile edges and large networks (both forms of the
background draw), rates on both sides of the window-wide draw's limit, windows of 2 to 16
steps, busy windows, active astrocytes, facilitation, and calls that split windows.  The
digests come from the library of commit 9485e4f with ASTROSIM_STEPPER=plain, the last one
with such an engine."""
import hashlib
import json
from pathlib import Path

import numpy as np
import pytest

import astrosimgpu_cuda_b200 as asg

pytestmark = pytest.mark.gpu

STATE = ("V", "w", "g_ex", "dg_ex", "g_in", "dg_in", "I_sic", "stp_x", "stp_u", "stp_t_last",
         "Ca", "IP3", "h", "sic_factor")
GOLDEN = Path(__file__).parent / "golden" / "window_states.json"

ACTIVE = {"SIC_th": 0.07, "w_a2n": 2.0, "sic_interval": 3}
BUSY = {"w_e": 40.0, "SIC_th": 0.0715, "stp_tau_fac": 30.0, "stp_U": 0.3}
SPLIT = (4, 1, 30, 7, 58)
LARGE = 48003  # neurons draw two to a thread

CASES = {}
for _n in (1, 5, 39, 41, 161, 321, 641, 2561, LARGE):
    CASES[f"size {_n}"] = ({}, SPLIT, dict(n_total=_n, seed=_n, neuron_drive_scale=1.2))
    CASES[f"active {_n}"] = (ACTIVE, SPLIT, dict(n_total=_n, seed=_n))
for _n in (700, LARGE):
    for _r in (0.0, 1.0, 12000.0, 39990.0, 40010.0, 150000.0, 310000.0):
        CASES[f"rate {_r:g} size {_n}"] = (
            {"exc_poiss_rate": _r, "inh_poiss_rate": 2500.0, "exc_poiss_weight": 0.02, "astro_poiss_rate": _r},
            (3, 17, 80), dict(n_total=_n, seed=3))
for _n in (1500, LARGE):
    for _dt, _sub in ((0.0625, 1), (0.1, 3), (0.5, 1)):
        CASES[f"dt {_dt:g} size {_n}"] = (
            {"e_t_ref": 1.3, "i_t_ref": 0.7, "sic_interval": 3, "noise_dt": 3 * _dt, "SIC_th": 0.07, "w_e": 40.0},
            (5, 3, 92), dict(n_total=_n, seed=9, dt=_dt, substeps=_sub))
    CASES[f"busy {_n}"] = (BUSY, (3, 97), dict(n_total=_n, seed=2, neuron_drive_scale=3.0))


def digest(case, precision):
    bio, chunks, kw = CASES[case]
    h = hashlib.sha256()
    with asg.Simulation(biology=bio, precision=precision, pre_ms=3.0, sim_ms=60.0, raster_steps=100, **kw) as sim:
        for c in chunks:
            sim.step(c)
        for name in STATE:
            h.update(np.ascontiguousarray(sim.state(name)).tobytes())
        h.update(np.ascontiguousarray(sim.spike_counts()).tobytes())
        h.update(sim.raster().tobytes())
        s = sim.summary()
        h.update(repr((s["spikes_total"], s["active_astro"], s["engaged_astro"])).encode())
    return h.hexdigest()[:16]


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("case", CASES)
def test_states(case, precision):
    assert digest(case, precision) == json.loads(GOLDEN.read_text())[case][precision]


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("variant", range(9))
@pytest.mark.parametrize("case", ["active 2561", "rate 12000 size 48003", f"busy {LARGE}"])
def test_every_variant(case, variant, precision, monkeypatch):
    monkeypatch.setenv("ASTROSIM_WINDOW_VARIANT", str(variant))
    assert digest(case, precision) == json.loads(GOLDEN.read_text())[case][precision]
