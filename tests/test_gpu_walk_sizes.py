"""The resident step kernels where their dealing of walkers and drawing of lengths can go wrong: fewer walkers than
lanes, one warp, one more, just past the walkers dealt without the counter, stop probabilities that end nearly every
walk at once or make one walk of a warp far longer than the others; paths of walks shorter and longer than the segments
they are gathered in; statistics.  Against the CPU oracle."""
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


@pytest.mark.parametrize("walkers,length", [(5003, n) for n in (1, 2, 31, 32, 33, 80)] + [(650003, n) for n in (9, 10, 14, 15, 16, 31, 32, 33)])
@pytest.mark.parametrize("wide", [True, False])
def test_walk_lengths(lt, require_gpu, graph, walkers, length, wide):
    import torch
    rp, col = graph
    V, W = len(rp) - 1, walkers
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


@pytest.mark.parametrize("degree", [63, 64, 80])
@pytest.mark.parametrize("layout", ["wide", "compact", "packed"])
def test_pagerank_shared_counters(lt, require_gpu, degree, layout):
    """More vertices at and around the least degree counted in shared memory than it has slots."""
    import torch
    V, W, L = 3001, 20011, 9
    rng = np.random.default_rng(degree)
    rp = (np.arange(V + 1, dtype=np.uint64) * np.uint64(degree))
    col = rng.integers(0, V, V * degree).astype(np.uint32)
    want, st = oracle.pagerank(rp, col, W, length=L, seed=77, start_mode=1)
    dev, p = "cuda", torch.cuda.current_stream().cuda_stream
    d_rp = torch.from_numpy(rp.view(np.int64)).to(dev)
    d_col = torch.from_numpy(col.view(np.int32)).to(dev)
    scratch = torch.zeros(lt.lib.lt_walk_scratch_bytes() // 8, dtype=torch.int64, device=dev)
    stats = torch.zeros(3, dtype=torch.int64, device=dev)
    tail = (scratch.data_ptr(), stats.data_ptr(), p)
    args = (V, 0, W, L, ctypes.c_float(0.85), 0, 77)
    if layout == "packed":
        rows = torch.empty(2 * (V + 1), dtype=torch.int32, device=dev)
        counts = torch.zeros(V, dtype=torch.int64, device=dev)
        lt.check(lt.lib.lt_rows_pack(d_rp.data_ptr(), rows.data_ptr(), V, p))
        lt.check(lt.lib.lt_walk_device_packed(1, 1, rows.data_ptr(), d_col.data_ptr(), *args, None, None, *tail))
        lt.check(lt.lib.lt_rows_counts(rows.data_ptr(), counts.data_ptr(), V, p))
    elif layout == "compact":
        rows = torch.from_numpy(rp.astype(np.uint32).view(np.int32)).to(dev)
        counts = torch.zeros(V, dtype=torch.int32, device=dev)
        lt.check(lt.lib.lt_walk_device_compact(1, 1, rows.data_ptr(), d_col.data_ptr(), *args, counts.data_ptr(), None, None, *tail))
    else:
        counts = torch.zeros(V, dtype=torch.int64, device=dev)
        lt.check(lt.lib.lt_walk_device(1, 1, d_rp.data_ptr(), d_col.data_ptr(), *args, counts.data_ptr(), None, None, *tail))
    assert (counts.cpu().numpy().astype(np.uint64) == want).all()
    assert stats.tolist() == [int(x) for x in st]


@pytest.mark.parametrize("walkers", [77824, 77825, 466944, 466945, 700417])  # edges of 2 and 3 CTAs per SM
@pytest.mark.parametrize("prob", [0.5, 0.15])
def test_ppr_ctas(lt, require_gpu, graph, walkers, prob):
    rp, col = graph
    e = lt.Engine(lt.Graph.from_csr(rp, col, 1 << 30), seed=55)
    want, _, st = oracle.ppr(rp, col, 3, walkers, prob=prob, seed=55)
    assert (e.ppr(3, walkers, prob) == want).all()
    s = e.stats()
    assert (s["updates"], s["moves"], s["teleports"]) == tuple(int(x) for x in st)
