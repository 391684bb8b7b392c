"""The walk kernels' remainder without 64-bit division at the divisors where its paths change and its bounds are
tightest: 1, powers of two and their neighbours, and both sides of 2^16 and 2^20 (folding up to 2^20, a corrected
quotient estimate above)."""
import ctypes

import numpy as np
import pytest


def _cases():
    d = [1, 2, 3, 5, 7, 65535, 65536, 65537, (1 << 20) - 1, 1 << 20, (1 << 20) + 1, (1 << 32) - 1]
    for b in range(2, 32):
        d += [(1 << b) - 1, 1 << b, (1 << b) + 1]
    rng = np.random.default_rng(11)
    d = np.array(sorted(set(d)), dtype=np.uint64)
    d = np.concatenate([d, rng.integers(1, (1 << 20) + 1, 3000, dtype=np.uint64)])
    top = np.uint64(0xFFFFFFFFFFFFFFFF)
    xs, ds = [], []
    for k in (0, 1, 2):  # around the largest multiples of d and of 2^32
        xs += [top - np.uint64(k) + np.zeros_like(d), (top // d) * d - np.uint64(k), d * np.uint64(0xFFFFFFFF) + np.uint64(k),
               (np.uint64(1) << np.uint64(32)) - np.uint64(k) + np.zeros_like(d)]
        ds += [d] * 4
    for _ in range(200):
        xs.append(rng.integers(0, top, len(d), dtype=np.uint64, endpoint=True))
        ds.append(d)
    return np.concatenate(xs), np.concatenate(ds)


def test_remainder_host(lt):
    x, d = _cases()
    out = np.empty_like(x)
    p = ctypes.POINTER(ctypes.c_uint64)
    lt.check(lt.lib.lt_mod_check(len(x), *(a.ctypes.data_as(p) for a in (x, d, out))))
    assert np.array_equal(out, x % d)


@pytest.mark.gpu
def test_remainder_device(lt, require_gpu):
    import torch
    x, d = _cases()
    tx, td = (torch.from_numpy(a.view(np.int64)).cuda() for a in (x, d))
    to = torch.empty_like(tx)
    lt.check(lt.lib.lt_mod_check_device(len(x), tx.data_ptr(), td.data_ptr(), to.data_ptr(),
                                        torch.cuda.current_stream().cuda_stream))
    assert np.array_equal(to.cpu().numpy().view(np.uint64), x % d)
