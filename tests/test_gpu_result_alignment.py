"""Results for addresses that are no multiple of their element's size: page-locked host arrays at an odd byte, device arrays
at an odd byte or at half an element."""
import ctypes

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
SEED, PROB = 3, 0.15


@pytest.fixture(scope="module")
def graph():
    return oracle.rmat(12, 1 << 15, seed=4)


def _pinned_at(lt, n, dtype, shift):
    return lt.pinned_empty((n + 1) * np.dtype(dtype).itemsize, np.uint8)[shift:shift + n * np.dtype(dtype).itemsize].view(dtype)


@pytest.mark.parametrize("shift", [0, 1, 4])
def test_counts(lt, require_gpu, graph, shift):
    rp, col = graph
    e = lt.Engine(lt.Graph.from_csr(rp, col, 1 << 30), seed=SEED)
    out = _pinned_at(lt, len(rp) - 1, np.uint64, shift)
    assert (e.ppr(1, 5000, PROB, out=out) == oracle.ppr(rp, col, 1, 5000, prob=PROB, seed=SEED)[0]).all()
    assert (e.pagerank(5000, length=5, out=out) == oracle.pagerank(rp, col, 5000, length=5, seed=SEED, start_mode=1)[0]).all()


def _check(rp, col, src, w, off, v, c):
    for q in range(len(src)):
        got = np.zeros(len(rp) - 1, np.uint64)
        a, b = int(off[q]), int(off[q + 1])
        got[v[a:b]] = c[a:b]
        assert (got == oracle.ppr(rp, col, int(src[q]), int(w[q]), prob=PROB, seed=SEED)[0]).all(), q


SRC, W = np.array([1, 2, 3], np.uint32), np.array([5000, 1, 12345], np.uint64)


@pytest.mark.parametrize("shifts", [(0, 0, 0), (1, 0, 0), (0, 2, 0), (0, 0, 3), (4, 1, 1)])
def test_batch_host(lt, require_gpu, graph, shifts):
    rp, col = graph
    e = lt.Engine(lt.Graph.from_csr(rp, col, 1 << 30), seed=SEED)
    n, total = len(SRC), int(W.sum())
    out = [_pinned_at(lt, k, t, s) for k, t, s in zip((n + 1, total, total), (np.uint64, np.uint32, np.uint32), shifts)]
    _check(rp, col, SRC, W, *e.ppr_batch(SRC, W, None, PROB, out=out))


@pytest.mark.parametrize("shifts", [(0, 0, 0), (1, 0, 0), (4, 0, 0), (0, 2, 0), (0, 0, 3), (4, 1, 1)])
def test_batch_device(lt, require_gpu, graph, shifts):
    import torch
    rp, col = graph
    e = lt.Engine(lt.Graph.from_csr(rp, col, 1 << 30), seed=SEED)
    n, total = len(SRC), int(W.sum())
    seeds = np.full(n, SEED, np.int64)
    d = [torch.from_numpy(a).cuda() for a in (SRC.view(np.int32), W.view(np.int64), seeds)]
    sizes = (8 * (n + 1), 4 * total, 4 * total)
    raw = [torch.full((k + 8,), 77, dtype=torch.uint8, device="cuda") for k in sizes]
    lt.check(lt.lib.lt_ppr_batch_device(e._h, n, *(x.data_ptr() for x in d), ctypes.c_float(PROB),
                                        *(r.data_ptr() + s for r, s in zip(raw, shifts)), total,
                                        torch.cuda.current_stream().cuda_stream))
    host = [r.cpu().numpy() for r in raw]
    for r, s, k in zip(host, shifts, sizes):
        assert (r[:s] == 77).all() and (r[s + k:] == 77).all()
    off, v, c = (r[s:s + k].copy().view(t) for r, s, k, t in zip(host, shifts, sizes, (np.uint64, np.uint32, np.uint32)))
    _check(rp, col, SRC, W, off, v, c)
