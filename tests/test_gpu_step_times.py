"""The time of the step kernels that a call reports does not depend on where its results go: the same kernels run, page-locked
or not, and only the way of the results differs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graph(lt, require_gpu):
    # 2^23 ids: 37 MB of counts, whose way over the host link takes several times as long as the walks below
    return lt.Graph.rmat(23, 1 << 25, seed=2, part_bytes=1 << 30)


def _least(call, e, key="step_kernel_ms"):
    t = []
    for _ in range(10):
        call()
        t.append(e.stats()[key])
    return min(t)


def test_step_time_of_a_run(lt, graph):
    e = lt.Engine(graph, seed=3)
    pinned, plain = lt.pinned_empty(graph.num_nodes), np.zeros(graph.num_nodes, np.uint64)
    for call in (lambda out: e.ppr(0, 20000, 0.3, out=out), lambda out: e.pagerank(20000, length=5, start=2, out=out)):
        a, b = (_least(lambda: call(out), e) for out in (pinned, plain))
        assert (pinned == plain).all()
        assert a < 1.3 * b and b < 1.3 * a


def test_step_time_of_a_batch(lt, require_gpu):
    # one hop to one of 512 vertices: some 2.6 million pairs, 21 MB, of as many short walks as they need
    rng = np.random.default_rng(1)
    V, n, each = 1 << 16, 8192, 512
    e = lt.Engine(lt.Graph.from_csr(512 * np.arange(V + 1, dtype=np.uint64), rng.integers(0, V, 512 * V).astype(np.uint32),
                                    1 << 30), seed=3)
    src, w = rng.integers(0, V, n).astype(np.uint32), np.full(n, each, np.uint64)
    kinds = [(np.uint64, n + 1), (np.uint32, n * each), (np.uint32, n * each)]
    pinned, plain = [lt.pinned_empty(k, t) for t, k in kinds], [np.zeros(k, t) for t, k in kinds]
    a, b = (_least(lambda: e.ppr_batch(src, w, None, 1.0, out=out), e) for out in (pinned, plain))
    assert (pinned[0] == plain[0]).all() and int(pinned[0][-1]) > 2 << 20
    assert a < 1.2 * b and b < 1.2 * a
