"""PageRank on both sides of 2^32 updates, up to which CTAs count hubs in 32-bit counters of their own (above, a call becomes
several launches, or one without such counters where the walks are long): 20 more walkers add their own updates, and no
vertex loses any."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length", [60, 4000])
def test_updates_beyond_32_bits(lt, require_gpu, length):
    import torch
    g = lt.Graph.rmat(14, 1 << 18, seed=5, part_bytes=1 << 30)
    rp, col = (torch.from_numpy(a.view(t)).cuda() for a, t in zip(g.csr_views(), ("int64", "int32")))
    V = g.num_nodes
    scratch = torch.zeros(lt.lib.lt_walk_scratch_bytes(), dtype=torch.uint8, device="cuda")
    last = ((1 << 32) - 1) // length
    counts, stats = [], []
    for walkers in (last, last + 1, last + 20):
        c, s = torch.zeros(V, dtype=torch.int64, device="cuda"), torch.zeros(3, dtype=torch.int64, device="cuda")
        lt.check(lt.lib.lt_walk_device(1, 1, rp.data_ptr(), col.data_ptr(), V, 0, walkers, length, ctypes.c_float(0.85), 0, 9,
                                       c.data_ptr(), None, None, scratch.data_ptr(), s.data_ptr(),
                                       torch.cuda.current_stream().cuda_stream))
        counts.append(c.cpu())
        stats.append(s.cpu().tolist())
        assert int(counts[-1].sum()) == walkers * length == stats[-1][0]
        assert stats[-1][1] + stats[-1][2] == walkers * (length - 1)
    for a, b, more in ((counts[0], counts[1], 1), (counts[1], counts[2], 19)):
        assert (b >= a).all() and int((b - a).sum()) == more * length
