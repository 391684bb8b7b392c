"""The resident step kernels where their dealing of walkers and drawing of lengths can go wrong: fewer walkers than
lanes, one warp, one more, just past the walkers dealt without the counter, stop probabilities that end nearly every
walk at once or make one walk of a warp far longer than the others, and statistics, against the CPU oracle."""
import ctypes

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graph():
    return oracle.rmat(13, 1 << 16, seed=9)


@pytest.mark.parametrize("walkers", [1, 31, 32, 33, 257, 38912, 38913, 311295, 311297])
@pytest.mark.parametrize("prob", [1.0, 0.5, 0.15, 0.02])
def test_ppr_walkers(lt, require_gpu, graph, walkers, prob):
    rp, col = graph
    e = lt.Engine(lt.Graph.from_csr(rp, col, 1 << 30), seed=123456789012345)
    want, _, st = oracle.ppr(rp, col, 2, walkers, prob=prob, seed=123456789012345)
    assert (e.ppr(2, walkers, prob) == want).all()
    s = e.stats()
    assert (s["updates"], s["moves"], s["teleports"]) == tuple(int(x) for x in st)


@pytest.mark.parametrize("walkers", [1, 33, 311296, 400001])
@pytest.mark.parametrize("alpha", [0.0, 0.3, 1.0])
@pytest.mark.parametrize("start", [1, 2])
def test_pagerank_walkers(lt, require_gpu, graph, walkers, alpha, start):
    rp, col = graph
    e = lt.Engine(lt.Graph.from_csr(rp, col, 1 << 30), seed=7)
    want, st = oracle.pagerank(rp, col, walkers, length=5, alpha=alpha, seed=7, start_mode=start)
    assert (e.pagerank(walkers, length=5, alpha=alpha, start=start) == want).all()
    s = e.stats()
    assert (s["updates"], s["moves"], s["teleports"]) == tuple(int(x) for x in st)


@pytest.mark.parametrize("length", [1, 2, 31, 32, 33, 80])
@pytest.mark.parametrize("wide", [True, False])
def test_walk_lengths(lt, require_gpu, graph, length, wide):
    import torch
    rp, col = graph
    V, W = len(rp) - 1, 5003
    rows = torch.from_numpy(rp.view(np.int64) if wide else rp.astype(np.uint32).view(np.int32)).cuda()
    d_col = torch.from_numpy(col.view(np.int32)).cuda()
    ep = torch.zeros(W, dtype=torch.int32, device="cuda")
    paths = torch.zeros(W * (length + 1) + 4, dtype=torch.int32, device="cuda")
    scratch = torch.zeros(lt.lib.lt_walk_scratch_bytes() // 8, dtype=torch.int64, device="cuda")
    stats = torch.zeros(3, dtype=torch.int64, device="cuda")
    call = lt.lib.lt_walk_device if wide else lt.lib.lt_walk_device_compact
    want_ep, want_pa, st = oracle.generic_walk(rp, col, W, length=length, start_mode=2, run=4, seed=31, paths=True)
    for off in (0, 1):  # the paths need not start on a 16-byte boundary
        stats.zero_()
        lt.check(call(2, 2, rows.data_ptr(), d_col.data_ptr(), V, 0, W, length, ctypes.c_float(0), 4, 31, None, ep.data_ptr(),
                      paths.data_ptr() + 4 * off, scratch.data_ptr(), stats.data_ptr(), torch.cuda.current_stream().cuda_stream))
        assert (ep.cpu().numpy().view(np.uint32) == want_ep).all()
        got = paths.cpu().numpy().view(np.uint32)
        assert (got[off:off + W * (length + 1)] == want_pa.ravel()).all() and (got[off + W * (length + 1):] == 0).all()
        assert stats.tolist() == [int(x) for x in st]
