"""What a call of few steps costs where the engine advances windows: it does the work of its
own steps.  The limits are ratios of device times of the same process, far from both what
the work asks for and what a window's work in every call takes."""
import statistics

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
