"""The prefetcher's kernels at the edges of their tiles: rows around a backward CTA's 256 threads and a warp, and the
policy's row kernels (one warp per partition, four per CTA) at partition counts on both sides of a CTA's edge."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 32, 33, 255, 256, 257, 513])
def test_backward_and_step(lt, require_gpu, n):
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, (n, oracle.MLP_IN)).astype(np.float32)
    y = rng.uniform(0, 1, n).astype(np.float32)
    p = (rng.standard_normal(oracle.MLP_PARAMS) * 0.3).astype(np.float32)
    pred, grad, loss, newp = lt.mlp_check(x, y, p, lr=0.05, momentum=0.9)
    wp, wg, wl = oracle.mlp_forward_backward(x, y, p)
    # FP32 against float64: the bounds of the other row counts
    np.testing.assert_allclose(pred, wp, rtol=1e-4, atol=1e-5)
    np.testing.assert_allclose(grad, wg, rtol=2e-3, atol=1e-6 + 1e-4 * np.abs(wg).max())
    assert abs(loss - wl) <= 1e-4 * max(1.0, wl)
    # fresh momentum: v = g, w -= lr v, one rounding of each
    np.testing.assert_allclose(newp, p - np.float32(0.05) * grad, rtol=1e-6, atol=1e-7)


@pytest.mark.parametrize("part_bytes", [16 << 10, 20 << 10, 33 << 10, 64 << 10])
def test_partition_rows(lt, require_gpu, part_bytes):
    rp, col = oracle.rmat(13, 1 << 17, seed=3)
    g = lt.Graph.from_csr(rp, col, part_bytes)
    share = -(-8 * len(rp) // part_bytes)
    e = lt.Engine(g, partitions=share + 3, seed=11, sched=lt.SCHED_LEARNED)
    for run in range(3):
        want, _, _ = oracle.ppr(rp, col, 1, 60000, prob=0.05, seed=11)
        assert (e.ppr(1, 60000, 0.05) == want).all()
    ps = e.policy_stats()
    assert ps["train_steps"] >= 1
    assert np.isfinite([ps["net_loss"], ps["baseline_loss"]]).all() and ps["baseline_loss"] >= 0
