"""What work costs away from whole windows of a single network: a call of few steps where the
engine advances windows, a batch that holds one large network.  The limits are ratios of
device times of the same process, far from both what the work asks for and what the
form that the test guards against takes."""
import statistics

import numpy as np
import pytest

import astrosimgpu_cuda_b200 as asg

pytestmark = pytest.mark.gpu


def median_ms(sim, steps, calls):
    out = []
    for _ in range(calls):
        sim.step(steps)
        out.append(sim.last_step_ms())
    return statistics.median(out)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_single_steps_of_a_delay_window(precision):
    """Delays of 20 steps run in windows of 16.  A single step has a sixteenth of a window's
    background draws and steps, and the same rows to walk: less than half of a window's time."""
    bio = {"d_e": 2.0, "d_i": 2.0, "d_a2n": 2.0}
    with asg.Simulation(biology=bio, n_total=200003, seed=3, pre_ms=2, sim_ms=100, precision=precision) as sim:
        sim.step(160)
        window = median_ms(sim, 16, 12)
        single = median_ms(sim, 1, 48)
    assert single < 0.5 * window, (single, window)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_a_batch_of_one_large_network(precision):
    """A batch delivers a large network's window and marks its active astrocytes' rows with as
    many blocks as the network needs: less than three times the network's own time."""
    kw = dict(n_total=200003, seed=3, pre_ms=2, sim_ms=100, precision=precision)
    bio = {"SIC_th": 0.07}  # every astrocyte active
    with asg.Simulation(biology=bio, **kw) as sim:
        sim.step(300)
        alone = median_ms(sim, 100, 3)
        states = [sim.state(k) for k in ("V", "I_sic", "Ca")]
    with asg.Ensemble([asg.default_config(**kw)], biology=[bio]) as ens:
        ens.step(300)
        batch = median_ms(ens, 100, 3)
        for k, a in zip(("V", "I_sic", "Ca"), states):
            np.testing.assert_array_equal(ens.state(0, k), a)
    assert batch < 3.0 * alone, (batch, alone)
