"""A batch whose tables do not fit the device is refused and leaves the engine as usable as before: the same batch is refused
again, and one that fits runs on buffers of its own."""
import ctypes

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("before", [False, True])
def test_batch_that_does_not_fit(lt, require_gpu, before):
    rp, col = oracle.rmat(12, 1 << 15, seed=4)
    e = lt.Engine(lt.Graph.from_csr(rp, col, 1 << 30), seed=3)

    def fits():
        off, v, c = e.ppr_batch([1, 9], [3000, 20], [5, 6], 0.15)
        for q, (s, w, k) in enumerate([(1, 3000, 5), (9, 20, 6)]):
            got = np.zeros(len(rp) - 1, np.uint64)
            got[v[int(off[q]):int(off[q + 1])]] = c[int(off[q]):int(off[q + 1])]
            assert (got == oracle.ppr(rp, col, s, w, prob=0.15, seed=k)[0]).all()

    u32, u64 = (ctypes.POINTER(t) for t in (ctypes.c_uint32, ctypes.c_uint64))
    src, walkers, off = np.zeros(1, np.uint32), np.array([1 << 38], np.uint64), np.zeros(2, np.uint64)
    out = np.zeros(1, np.uint32)  # never reached: 2 TiB of tables come first
    if before:
        fits()
    for _ in range(2):
        st = lt.lib.lt_ppr_batch(e._h, 1, src.ctypes.data_as(u32), walkers.ctypes.data_as(u64), None, 0.15,
                                 off.ctypes.data_as(u64), out.ctypes.data_as(u32), out.ctypes.data_as(u32), 1 << 38)
        with pytest.raises(lt.LTError, match="LT_ERR_NOMEM"):
            lt.check(st)
    fits()
