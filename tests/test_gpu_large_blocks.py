"""Block sizes up to the largest that a configuration may ask for, in both engines and
precisions, and networks of different window lengths stepped by several threads at once: the
block size never changes a result."""
import threading

import numpy as np
import pytest

import astrosimgpu_cuda_b200 as asg

pytestmark = pytest.mark.gpu

STATES = ("V", "w", "g_ex", "g_in", "I_sic", "Ca", "IP3", "sic_factor")


def states(chunks, biology=None, **kw):
    with asg.Simulation(biology=biology, n_total=3000, seed=8, pre_ms=2, sim_ms=200, **kw) as sim:
        for c in chunks:
            sim.step(c)
        return [sim.state(k) for k in STATES]


def test_threads_with_different_windows():
    """Windows of 10 and 16 steps of the same kernel need different amounts of shared memory;
    networks stepped by different threads must not set each other's limit."""
    chunks = (10,) * 150
    runs = [dict(block=1024, dt=dt, precision="fp64") for dt in (0.1, 0.0625)] * 2
    want = {dt: states(chunks, dt=dt, precision="fp64") for dt in (0.1, 0.0625)}
    got, errors = [None] * len(runs), []

    def work(i):
        try:
            got[i] = states(chunks, **runs[i])
        except Exception as e:  # reported below, in the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(runs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for run, result in zip(runs, got):
        for a, b in zip(result, want[run["dt"]]):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("block", [736, 768, 1024])
def test_delay_windows(block, precision):
    """Delays that the windowed engine does not take: the registers of the FP64 form bound its
    blocks below the largest that a configuration may ask for."""
    bio = {"w_e": 25.0, "SIC_th": 0.0715, "d_e": 0.6, "d_i": 1.6, "d_a2n": 1.0}
    chunks = (3, 47, 50)
    for a, b in zip(states(chunks, bio, block=block, precision=precision), states(chunks, bio, precision=precision)):
        np.testing.assert_array_equal(a, b)
