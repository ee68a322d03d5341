"""The window-wide background draw against the per-step draw it replaces, count by count, on
the host (no GPU): tests/poisson_window_check.cpp.  Rates run from 1e-20 events per step,
where e^-lambda rounds to 1 and no step has an event, over the default's 0.3 to both sides
of the window-wide form's limit of 4."""
import os
import re
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = tmp_path_factory.mktemp("poisson") / "poisson_window_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", str(exe),
                    os.path.join(HERE, "poisson_window_check.cpp")], check=True)
    return str(exe)


@pytest.mark.parametrize("lam", [0.0, 1e-20, 1e-17, 1.2e-16, 1e-12, 1e-10, 2.4e-10, 1e-8, 1e-4, 0.01, 0.3, 1.0, 2.5,
                                 3.999, 4.0, 4.001, 12.0, 45.0])
def test_counts_are_the_per_step_draws(checker, lam):
    r = subprocess.run([checker, repr(lam), "12"], capture_output=True, text=True, timeout=300)
    m = re.search(r"checked (\d+) wrong (\d+) exact (\d+) events (\d+) past (\d+)", r.stdout)
    assert m, r.stdout + r.stderr
    checked, wrong, exact, events, past = (int(x) for x in m.groups())
    assert r.returncode == 0 and wrong == 0, r.stdout
    assert checked > 400000
    if lam == 0.0:
        assert exact == 0 and events == 0
    elif lam > 4.0:
        assert exact == checked
    else:
        assert exact < checked / 100  # the others are compared count by count
    if lam >= 0.01:
        assert events > 1000


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("delay", [1.0, 0.7])
def test_rates_too_small_for_an_event(delay, precision):
    """Both engines: a rate of 1e-13 Hz has no event in any step a run can have, so every
    state equals that of a run without background."""
    import astrosimgpu_cuda_b200 as asg

    out = []
    for rate in (0.0, 1e-13):
        bio = {"exc_poiss_rate": rate, "inh_poiss_rate": rate, "astro_poiss_rate": rate, "d_e": delay}
        with asg.Simulation(biology=bio, n_total=700, seed=4, pre_ms=2, sim_ms=20, precision=precision) as sim:
            sim.step(200)
            out.append([sim.state(k) for k in ("V", "w", "g_ex", "g_in", "Ca", "IP3")])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
