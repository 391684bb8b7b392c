"""Bursts of queries: admitted together and in several admissions (slots or pool short), several per partition
chunk, of one walker and of more than a chunk, finishing together and apart; each result equals the oracle's alone."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slots,table,pool", [(64, 1 << 20, 1 << 18), (5, 1 << 20, 1 << 18), (64, 1 << 20, 1 << 16)])
@pytest.mark.parametrize("sched", [0, 2, 4])
def test_bursts(lt, require_gpu, slots, table, pool, sched):
    rp, col = oracle.rmat(14, 1 << 18, seed=6)
    g = lt.Graph.from_csr(rp, col, 32 << 10)
    e = lt.Engine(g, partitions=-(-8 * len(rp) // (32 << 10)) + 6, batch=pool, seed=3, sched=sched)
    srv = lt.Server(e, max_active=slots, table_slots=table, prob=0.2)
    rng = np.random.default_rng(sched * 100 + slots)
    for burst in (1, 17, 40):
        w = np.concatenate([[1, 2, 8191, 8193, 12000], rng.integers(1, 3000, 40)])[:burst]
        src = rng.integers(0, min(50, len(rp) - 1), burst)  # many of one partition
        sd = rng.integers(1, 1 << 62, burst)
        tickets = [srv.submit(int(a), int(b), int(c)) for a, b, c in zip(src, w, sd)]
        left, rounds = set(tickets), 0
        while left:
            srv.step()
            left -= set(srv.finished())
            rounds += 1
            assert rounds < 20000
        for t, a, b, c in zip(tickets, src, w, sd):
            got, _ = srv.result(t)
            counts, _, _ = oracle.ppr(rp, col, int(a), int(b), prob=0.2, seed=int(c))
            nz = np.nonzero(counts)[0]
            assert got == dict(zip(nz.tolist(), counts[nz].tolist()))
    srv.close()
    e.close()


@pytest.mark.parametrize("part_bytes", [2000, 16 << 10, 120 << 10])  # 487, 59 and 8 slices of odd lengths at any word
@pytest.mark.parametrize("sched", [3, 4])
def test_small_loads(lt, require_gpu, part_bytes, sched):
    rng = np.random.default_rng(12)
    V = 30011
    deg = rng.integers(0, 13, V)
    rp = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint64)
    col = rng.integers(0, V, int(rp[-1])).astype(np.uint32)
    g = lt.Graph.from_csr(rp, col, part_bytes)
    share = -(-8 * len(rp) // part_bytes)
    e = lt.Engine(g, partitions=min(g.num_partitions - 1, share + max(1, g.num_partitions // 2)), batch=1 << 18, seed=3,
                  sched=sched, zerocopy_threshold=1)
    srv = lt.Server(e, max_active=32, table_slots=1 << 20, prob=0.1)
    q = [(int(s), 3000 + 7 * k, 100 + k) for k, s in enumerate(rng.integers(0, V, 20))]
    tickets = [srv.submit(*x) for x in q]
    left, rounds = set(tickets), 0
    while left:
        srv.step()
        left -= set(srv.finished())
        rounds += 1
        assert rounds < 20000
    for t, (a, b, c) in zip(tickets, q):
        got, _ = srv.result(t)
        counts, _, _ = oracle.ppr(rp, col, a, b, prob=0.1, seed=c)
        nz = np.nonzero(counts)[0]
        assert got == dict(zip(nz.tolist(), counts[nz].tolist()))
    assert e.stats()["partition_loads"] > 1
    srv.close()
    e.close()
