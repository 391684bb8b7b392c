"""The out-of-core step kernel where its tables and its dealing of walkers change: partition counts at which column
addresses and then the whole partition table leave shared memory, few and many walkers, starts whose walkers are created
for many partitions in one pass, in part, or over several passes; against the CPU oracle."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def regular():
    """Every vertex has 8 out-edges, one in ten has none."""
    rng = np.random.default_rng(8)
    V = 20011
    deg = np.where(rng.random(V) < 0.1, 0, 8)
    rp = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint64)
    return rp, rng.integers(0, V, int(rp[-1])).astype(np.uint32)


@pytest.fixture(scope="module")
def skewed():
    return oracle.rmat(14, 1 << 18, seed=6)


@pytest.mark.parametrize("part_bytes", [200, 400, 1000, 64 << 10])  # 4 514, 2 008, 757 and 12 partitions
@pytest.mark.parametrize("sched", [0, 4])
@pytest.mark.parametrize("index", [True, False])
def test_partition_counts(lt, require_gpu, regular, part_bytes, sched, index):
    rp, col = regular
    V, W = len(rp) - 1, 3001 if sched == 0 else 30011
    g = lt.Graph.from_csr(rp, col, part_bytes)
    share = -(-8 * len(rp) // part_bytes) if index else 0
    e = lt.Engine(g, partitions=min(g.num_partitions - 1, share + max(2, g.num_partitions // 5)), seed=9, sched=sched,
                  resident_index=index)
    want, _, st = oracle.ppr(rp, col, 5, W, prob=0.2, seed=9)
    assert (e.ppr(5, W, 0.2) == want).all()
    s = e.stats()
    assert (s["updates"], s["moves"]) == (int(st[0]), int(st[1]))
    if sched:
        want, st = oracle.pagerank(rp, col, W, length=6, seed=9, start_mode=2)
        assert (e.pagerank(W, length=6, start=2) == want).all()
        s = e.stats()
        assert (s["updates"], s["moves"], s["teleports"]) == tuple(int(x) for x in st)


@pytest.mark.parametrize("walkers", [1, 33, 5000, 10961, 10962, 40000, 250007])
@pytest.mark.parametrize("pool", [0, 65536])
@pytest.mark.parametrize("start", [1, 2])
def test_created_walkers(lt, require_gpu, skewed, walkers, pool, start):
    rp, col = skewed
    g = lt.Graph.from_csr(rp, col, 32 << 10)
    share = -(-8 * len(rp) // (32 << 10))
    for sched in (3, 4):
        e = lt.Engine(g, partitions=share + 4, batch=pool, seed=77, sched=sched)
        want, st = oracle.pagerank(rp, col, walkers, length=5, runs=2, seed=77, start_mode=start)
        assert (e.pagerank(walkers, length=5, runs=2, start=start) == want).all()
        s = e.stats()
        assert (s["updates"], s["moves"], s["teleports"]) == tuple(int(x) for x in st)
        ep, pa, _ = oracle.generic_walk(rp, col, walkers, length=4, start_mode=start, run=1, seed=77, paths=True)
        got_ep, got_pa = e.walk(walkers, length=4, run=1, start=start, paths=True)
        assert (got_ep == ep).all() and (got_pa == pa.ravel()).all()


@pytest.mark.parametrize("walkers", [1, 31, 4097, 100003])
@pytest.mark.parametrize("prob", [0.9, 0.15, 0.03])
def test_ppr_lengths(lt, require_gpu, skewed, walkers, prob):
    rp, col = skewed
    g = lt.Graph.from_csr(rp, col, 32 << 10)
    e = lt.Engine(g, partitions=-(-8 * len(rp) // (32 << 10)) + 5, batch=1 << 15, seed=12345678901, sched=4)
    want, _, st = oracle.ppr(rp, col, 0, walkers, prob=prob, seed=12345678901)
    assert (e.ppr(0, walkers, prob) == want).all()
    assert e.stats()["moves"] == int(st[1])


@pytest.mark.parametrize("part_bytes", [240, 1000, 64 << 10])  # 3 611 partitions (tiles of 4096), 757 and 12
@pytest.mark.parametrize("walkers", [1023, 1025, 160003, 2600003])  # one tile to several of the largest per CTA
@pytest.mark.parametrize("items", [0, 8])
def test_bucket_tiles(lt, require_gpu, regular, part_bytes, walkers, items):
    rp, col = regular
    g = lt.Graph.from_csr(rp, col, part_bytes)
    share = -(-8 * len(rp) // part_bytes)
    e = lt.Engine(g, partitions=min(g.num_partitions - 1, share + 2), seed=9, sched=3, bucket_items=items)
    want, st = oracle.pagerank(rp, col, walkers, length=4, seed=9, start_mode=2)
    assert (e.pagerank(walkers, length=4, start=2) == want).all()
    s = e.stats()
    assert (s["updates"], s["moves"], s["teleports"]) == tuple(int(x) for x in st)


@pytest.mark.parametrize("part_bytes", [2000, 16 << 10, 120 << 10])  # 487, 59 and 8 slices of odd lengths at any word
@pytest.mark.parametrize("pipeline", [True, False])
@pytest.mark.parametrize("sched", [3, 4])
def test_small_loads(lt, require_gpu, part_bytes, pipeline, sched):
    rng = np.random.default_rng(12)
    V = 30011
    deg = rng.integers(0, 13, V)
    rp = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint64)
    col = rng.integers(0, V, int(rp[-1])).astype(np.uint32)
    g = lt.Graph.from_csr(rp, col, part_bytes)
    share = -(-8 * len(rp) // part_bytes)
    e = lt.Engine(g, partitions=min(g.num_partitions - 1, share + max(1, g.num_partitions // 2)), seed=3, sched=sched,
                  pipeline=pipeline, load_factor=1)
    for run in range(2):
        want, _, st = oracle.ppr(rp, col, 7, 120011, prob=0.1, seed=3)
        assert (e.ppr(7, 120011, 0.1) == want).all()
        s = e.stats()
        assert (s["updates"], s["moves"]) == (int(st[0]), int(st[1]))
