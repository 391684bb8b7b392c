"""Kernel times of out-of-core runs, kept by the kernels themselves: every kind of pass (plain and wave runs, plans made
on the device and on the host, split launches) leaves times that fit into the run's own, none of them from an earlier run."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sched", [0, 4])
@pytest.mark.parametrize("host_plan", [False, True])
@pytest.mark.parametrize("split", [False, True])
def test_times(lt, require_gpu, sched, host_plan, split):
    g = lt.Graph.rmat(15, 1 << 19, seed=2, part_bytes=64 << 10)
    share = -(-8 * g.num_nodes // (64 << 10))
    e = lt.Engine(g, partitions=share + 6, seed=5, sched=sched, host_plan=host_plan, split=split)
    for walkers in (200000, 2000):  # a long run, then a short one
        e.ppr(0, walkers, 0.15)
        s = e.stats()
        assert s["handoffs"] > 0 and s["partition_loads"] >= 0
        assert 0 < s["step_kernel_ms"] and 0 < s["bucket_ms"] < s["running_ms"]
        assert abs(s["step_kernel_ms"] - s["computing_ms"] - s["zerocopy_ms"]) < 1e-6 * s["step_kernel_ms"]
        # passes follow one another; the two kernels of a split launch overlap
        assert s["computing_ms"] < s["running_ms"] and s["zerocopy_ms"] < s["running_ms"]
        assert (s["computing_calls"] > 0) == (s["computing_ms"] > 0)
        assert (s["zerocopy_calls"] > 0) == (s["zerocopy_ms"] > 0)
