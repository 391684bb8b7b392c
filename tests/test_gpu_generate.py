"""The GPU RMAT generator against the CPU restatement where its kernels' edges lie: graphs with fewer ids than the
shared-memory counters, edge counts around one warp's share, sparse rows (many empty ones between two edges) and rows
longer than several warps' shares."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale,edges", [(1, 1), (1, 1023), (3, 511), (8, 512), (11, 513), (12, 40009), (13, 65536),
                                         (16, 100), (18, 5000), (20, 300001), (9, 1 << 20)])
@pytest.mark.parametrize("seed", [1, 0xABCDEF0123456789])
def test_rmat_edges(lt, require_gpu, scale, edges, seed):
    g = lt.Graph.rmat(scale, edges, seed=seed, part_bytes=1 << 30)
    rp, col = g.csr()
    want_rp, want_col = oracle.rmat(scale, edges, seed=seed)
    assert np.array_equal(rp, want_rp) and np.array_equal(col, want_col)


@pytest.mark.parametrize("probs", [(0.25, 0.25, 0.25, 0.25), (0.9, 0.05, 0.04, 0.01), (0.1, 0.0, 0.0, 0.9)])
def test_rmat_probabilities(lt, require_gpu, probs):
    a, b, c, d = probs
    g = lt.Graph.rmat(14, 70001, seed=5, part_bytes=1 << 30, a=a, b=b, c=c, d=d)
    rp, col = g.csr()
    want_rp, want_col = oracle.rmat(14, 70001, seed=5, a=a, b=b, c=c, d=d)
    assert np.array_equal(rp, want_rp) and np.array_equal(col, want_col)
