"""The launches a batch reports: prepare, clear, walk, count, compact, offsets, and the scan of the chunks' counts (by one CTA
up to 32 768 chunks of 4096 table slots, by three kernels above)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("walkers,launches", [(100, 7), (1 << 22, 7), (1 << 26, 9)])
def test_launches(lt, require_gpu, walkers, launches):
    e = lt.Engine(lt.Graph.rmat(12, 1 << 15, seed=2, part_bytes=1 << 30), seed=3)
    out = [lt.pinned_empty(n, t) for n, t in ((3, np.uint64), (walkers + 1, np.uint32), (walkers + 1, np.uint32))]
    off, v, c = e.ppr_batch([1, 2], [walkers, 1], None, 0.9, out=out)
    assert int(c.sum(dtype=np.uint64)) == walkers + 1
    assert e.stats()["kernel_launches"] == launches
