"""Out-of-core engines of different partition counts alive at the same time: the step kernel's shared memory depends on the
partition count (most at 1 536, less just above), and its limit belongs to the kernel, not to the engine."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def regular():
    """4 out-edges a vertex: 24 bytes each in a partition, and 8 for the partition."""
    V = 30011
    return 4 * np.arange(V + 1, dtype=np.uint64), np.random.default_rng(3).integers(0, V, 4 * V).astype(np.uint32)


# vertices a partition: 1 501 and 698 partitions, 1 112 and 639, 1 501 and 1 580, 3 752 and 1 501, 20 and 1 501
@pytest.mark.parametrize("per", [(20, 43), (43, 20), (27, 47), (20, 19), (8, 20), (1501, 20)])
def test_engines_of_two_partition_counts(lt, require_gpu, regular, per):
    rp, col = regular
    engines = []
    for n in per:
        g = lt.Graph.from_csr(rp, col, 24 * n + 8)
        assert g.num_partitions == -(-(len(rp) - 1) // n)
        share = -(-8 * len(rp) // (24 * n + 8))
        engines.append(lt.Engine(g, partitions=min(g.num_partitions - 1, share + max(2, g.num_partitions // 5)), seed=4,
                                 sched=4))
    ppr, _, _ = oracle.ppr(rp, col, 5, 20011, prob=0.2, seed=4)
    pr, _ = oracle.pagerank(rp, col, 20011, length=5, seed=4, start_mode=2)
    ep, _, _ = oracle.generic_walk(rp, col, 20011, length=4, start_mode=2, run=0, seed=4)
    for _ in range(2):
        for e in engines:
            assert (e.ppr(5, 20011, 0.2) == ppr).all()
            assert (e.pagerank(20011, length=5, start=2) == pr).all()
            assert (e.walk(20011, length=4, start=2)[0] == ep).all()
