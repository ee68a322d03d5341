"""Edges of the window kernels' tiles and of the background draws: network sizes around
one and two tiles of every block size (so that blocks and warps are partly
empty), background rates around the limits of the window-wide
draw, and the long windows of small steps.  The per-step path draws and rounds every step
by itself, and every result must equal it bit for bit."""
import numpy as np
import pytest

import astrosimgpu_cuda_b200 as asg

pytestmark = pytest.mark.gpu

STATES = ("V", "w", "g_ex", "dg_ex", "g_in", "dg_in", "I_sic", "stp_x", "stp_u", "stp_t_last", "Ca", "IP3", "h",
          "sic_factor")


def results(monkeypatch, stepper, chunks, biology, **kw):
    monkeypatch.setenv("ASTROSIM_STEPPER", stepper)
    with asg.Simulation(biology=biology, **kw) as sim:
        for c in chunks:
            sim.step(c)
        out = {k: sim.state(k) for k in STATES}
        out["counts"] = sim.spike_counts()
        out["engaged"] = sim.summary()["engaged_astro"]
    return out


def check(monkeypatch, chunks, biology=None, **kw):
    ref = results(monkeypatch, "plain", chunks, biology, **kw)
    got = results(monkeypatch, "auto", chunks, biology, **kw)
    for k in ref:
        np.testing.assert_array_equal(got[k], ref[k], err_msg=k)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("n_total", [1, 2, 5, 39, 40, 41, 79, 81, 160, 161, 319, 321, 640, 641, 1281, 2561])
def test_sizes_around_the_tiles(monkeypatch, n_total, precision):
    """0.8 n_total excitatory cells: 31-33, 63-65, 128, 129, 255-257, 512, 513, 1025, 2049 of them."""
    for variant in (0, 2, 3, 6, 8):
        monkeypatch.setenv("ASTROSIM_WINDOW_VARIANT", str(variant))
        check(monkeypatch, (4, 30, 87), n_total=n_total, seed=n_total, pre_ms=3, sim_ms=9, precision=precision,
              neuron_drive_scale=1.2)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("rate", [0.0, 1.0, 39990.0, 40010.0, 150000.0, 310000.0])
def test_background_rates(monkeypatch, rate, precision):
    """No background, almost none, lambda on both sides of the window-wide draw's limit (4 per
    step), counts past its four bits, and the normal approximation (lambda > 30)."""
    bio = {"exc_poiss_rate": rate, "inh_poiss_rate": 2500.0, "exc_poiss_weight": 0.02, "astro_poiss_rate": rate}
    check(monkeypatch, (3, 17, 200), bio, n_total=700, seed=3, pre_ms=2, sim_ms=20, precision=precision)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("dt,substeps", [(0.0625, 1), (0.1, 3), (0.5, 1)])
def test_window_lengths_and_refractory_cells(monkeypatch, dt, substeps, precision):
    """Windows of 16, 10 and 2 steps, clamped (refractory) steps, a SIC refresh every third
    step and a noise index that changes inside the window."""
    bio = {"e_t_ref": 1.3, "i_t_ref": 0.7, "sic_interval": 3, "noise_dt": 3 * dt, "SIC_th": 0.07, "w_e": 40.0}
    check(monkeypatch, (5, 3, 150), bio, n_total=1500, seed=9, pre_ms=2, sim_ms=20, dt=dt, substeps=substeps,
          precision=precision)
