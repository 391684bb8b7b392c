"""Batched PPR where a warp's pools, the gathered endpoints and the table chunks begin and end: queries without walkers,
of one walker, of one more or less than a pool or a chunk holds, few and many of them; results into page-locked memory,
fresh arrays and device buffers."""
import ctypes

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graph():
    return oracle.rmat(12, 1 << 15, seed=4)


def _check(rp, col, src, w, seeds, prob, off, v, c):
    assert off[0] == 0
    for q in range(len(src)):
        a, b = int(off[q]), int(off[q + 1])
        want, _, _ = oracle.ppr(rp, col, int(src[q]), int(w[q]), prob=prob, seed=int(seeds[q]))
        got = np.zeros(len(rp) - 1, np.uint64)
        np.add.at(got, v[a:b], c[a:b].astype(np.uint64))
        assert len(np.unique(v[a:b])) == b - a and (got == want).all(), q


SIZES = {"one": [1], "zeros": [0, 3, 0, 0, 17, 0], "pool": [255, 256, 257, 15, 16, 17, 31, 33, 511, 513],
         "chunk": [1023, 1024, 1025, 2047, 2048, 2049, 4095, 4097], "tiny": [1] * 700 + [2, 0, 5], "large": [300001, 7, 40000]}


@pytest.mark.parametrize("sizes", sorted(SIZES))
@pytest.mark.parametrize("prob", [0.15, 0.9])
def test_batch_sizes(lt, require_gpu, graph, sizes, prob):
    rp, col = graph
    w = np.array(SIZES[sizes], np.uint64)
    n, total = len(w), int(w.sum())
    rng = np.random.default_rng(n)
    src = rng.integers(0, len(rp) - 1, n).astype(np.uint32)
    seeds = rng.integers(1, 1 << 62, n, dtype=np.uint64)
    e = lt.Engine(lt.Graph.from_csr(rp, col, 1 << 30), seed=3)
    _check(rp, col, src, w, seeds, prob, *e.ppr_batch(src, w, seeds, prob))
    s = e.stats()
    assert s["updates"] == s["moves"] + total
    out = (lt.pinned_empty(n + 1, np.uint64), lt.pinned_empty(total, np.uint32), lt.pinned_empty(total, np.uint32))
    _check(rp, col, src, w, seeds, prob, *e.ppr_batch(src, w, seeds, prob, out=out))


def test_batch_device_buffers(lt, require_gpu, graph):
    import torch
    rp, col = graph
    w = np.array([5000, 0, 1, 12345], np.uint64)
    src, seeds = np.array([1, 2, 3, 4], np.uint32), np.array([9, 8, 7, 6], np.uint64)
    n, total = len(w), int(w.sum())
    e = lt.Engine(lt.Graph.from_csr(rp, col, 1 << 30), seed=3)
    d = [torch.from_numpy(a).cuda() for a in (src.view(np.int32), w.view(np.int64), seeds.view(np.int64))]
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    v, c = (torch.full((total + 3,), -7, dtype=torch.int32, device="cuda") for _ in range(2))
    for _ in range(2):
        lt.check(lt.lib.lt_ppr_batch_device(e._h, n, *(x.data_ptr() for x in d), ctypes.c_float(0.15), off.data_ptr(), v.data_ptr(),
                                            c.data_ptr(), total, torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        _check(rp, col, src, w, seeds, 0.15, off.cpu().numpy(), v.cpu().numpy().view(np.uint32), c.cpu().numpy().view(np.uint32))
    assert (v[total:] == -7).all() and (c[total:] == -7).all()
