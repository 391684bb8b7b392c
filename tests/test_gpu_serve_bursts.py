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
