"""What a rank of a sharded network launches per window: the window, and one push that also
draws the next window's background events (besides the packing for the other ranks).  Calls
that stop and go on draw each window's events once and give the unsplit run's states."""
import numpy as np
import pytest

from astrosimgpu_cuda_b200.shard import ShardGroup

pytestmark = pytest.mark.gpu


def kernels(run):
    """The kernels that `run` launches, by name."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    torch.cuda.init()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        run()
        torch.cuda.synchronize()
    return [e.name for e in prof.events() if "astrosim::" in e.name]  # the others: API calls, copies


def test_launches_per_window():
    with ShardGroup(world=2, n_total=3000, seed=3, pre_ms=2, sim_ms=60) as g:
        g.step(100)
        names = kernels(lambda: g.step(200))

    def count(part):
        return sum(part in n for n in names)

    assert count("shard_window_kernel") == 40  # 20 windows of two ranks
    assert count("shard_push_kernel") in (40, 42)  # and the draws of the call's first window
    assert sum(count(part) for part in ("shard_window", "shard_push", "pack_", "import_")) == len(names)


@pytest.mark.parametrize("world", [1, 2, 3])
def test_split_calls(world):
    out = []
    for chunks in ((200,), (10, 10, 50, 20, 110)):
        with ShardGroup(world=world, n_total=3000, seed=3, pre_ms=2, sim_ms=60, biology={"w_e": 25.0}) as g:
            for c in chunks:
                g.step(c)
            out.append([g.state(k) for k in ("V", "w", "g_ex", "g_in", "I_sic", "Ca", "IP3")])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
