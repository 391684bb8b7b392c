"""Batches of one engine enqueued one after another without a wait between them: on two streams, on a stream and then from
host arrays, and with buffers that have to grow while the batch before is still running."""
import ctypes

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graph():
    return oracle.rmat(16, 1 << 20, seed=4)


class _Batch:
    """Queries and result arrays on the device, the latter in front of a few words that stay as they are."""

    def __init__(self, torch, V, n, walkers, seed):
        rng = np.random.default_rng(seed)
        self.src, self.w = rng.integers(0, V, n).astype(np.uint32), np.full(n, walkers, np.uint64)
        self.seeds = rng.integers(1, 1 << 62, n, dtype=np.uint64)
        self.total = n * walkers
        self.dev = [torch.from_numpy(a).cuda() for a in (self.src.view(np.int32), self.w.view(np.int64), self.seeds.view(np.int64))]
        self.off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
        self.out = [torch.full((self.total + 1000,), -7, dtype=torch.int32, device="cuda") for _ in range(2)]

    def launch(self, lt, e, stream):
        lt.check(lt.lib.lt_ppr_batch_device(e._h, len(self.src), *(x.data_ptr() for x in self.dev), ctypes.c_float(0.15),
                                            self.off.data_ptr(), *(x.data_ptr() for x in self.out), self.total, stream))

    def check(self, rp, col):
        off, (v, c) = self.off.cpu().numpy(), (x.cpu().numpy() for x in self.out)
        assert (v[self.total:] == -7).all() and (c[self.total:] == -7).all()
        _check(rp, col, self, off, v, c)


def _check(rp, col, b, off, v, c):
    for q in range(0, len(b.src), max(1, len(b.src) // 3)):
        i, j = int(off[q]), int(off[q + 1])
        want, _, _ = oracle.ppr(rp, col, int(b.src[q]), int(b.w[q]), prob=0.15, seed=int(b.seeds[q]))
        got = np.zeros(len(rp) - 1, np.uint64)
        np.add.at(got, v[i:j], c[i:j].astype(np.uint64))
        assert (got == want).all(), q


@pytest.mark.parametrize("grow", [False, True])
def test_two_streams(lt, require_gpu, graph, grow):
    import torch
    rp, col = graph
    V = len(rp) - 1
    e = lt.Engine(lt.Graph.from_csr(rp, col, 1 << 30), seed=3)
    streams = [torch.cuda.Stream() for _ in range(2)]
    large, small = _Batch(torch, V, 200, 20000, 1), _Batch(torch, V, 3, 50, 2)
    torch.cuda.synchronize()
    order = [small, large] if grow else [large, small]
    for k in range(4):
        order[k % 2].launch(lt, e, streams[k % 2].cuda_stream)
    torch.cuda.synchronize()
    for b in order:
        b.check(rp, col)


@pytest.mark.parametrize("seeds", [True, False])
def test_stream_then_host(lt, require_gpu, graph, seeds):
    import torch
    rp, col = graph
    V = len(rp) - 1
    e = lt.Engine(lt.Graph.from_csr(rp, col, 1 << 30), seed=3)
    stream = torch.cuda.Stream()
    large, host = _Batch(torch, V, 200, 20000, 1), _Batch(torch, V, 5, 70, 2)
    if not seeds:
        host.seeds[:] = 3
    torch.cuda.synchronize()
    for _ in range(2):
        large.launch(lt, e, stream.cuda_stream)
        _check(rp, col, host, *e.ppr_batch(host.src, host.w, host.seeds if seeds else None, 0.15))
        torch.cuda.synchronize()
        large.check(rp, col)
