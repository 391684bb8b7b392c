"""The least PPR stop probability, 2^-26: below it walk lengths do not fit their 32 bits, and below 2^-53 no draw would ever
end a walk.  Every entry point refuses smaller ones before it launches anything."""
import ctypes
import struct

import numpy as np
import pytest

LEAST = 2.0 ** -26
SMALL = [1e-17, 2.0 ** -53, 2.0 ** -27, float(np.nextafter(np.float32(LEAST), np.float32(0)))]


def _walk_device(lt, prob, app=0):
    # no walkers: the arguments are checked, nothing is launched
    return lt.lib.lt_walk_device(app, 0, 256, 256, 10, 0, 0, 4, ctypes.c_float(prob), 0, 1, 256, None, None, 256, None, None)


@pytest.mark.parametrize("prob", SMALL + [0.0, -0.5, 1.5, float("nan")])
def test_refused_step_kernel(lt, prob):
    with pytest.raises(lt.LTError, match="LT_ERR_INVALID.*stop probability"):
        lt.check(_walk_device(lt, prob))
    lt.check(_walk_device(lt, prob, app=2))  # a generic walk has none


@pytest.mark.parametrize("prob", [LEAST, 1e-6, 0.15, 1.0])
def test_taken_step_kernel(lt, prob):
    lt.check(_walk_device(lt, prob))


@pytest.mark.parametrize("prob,ok", [(p, False) for p in SMALL] + [(LEAST, True), (0.15, True)])
def test_checkpoint_header(lt, tmp_path, prob, ok):
    f = tmp_path / "c"
    f.write_bytes(b"LTCKPT01" + struct.pack("<I", 2) + struct.pack("<8I", 0, 0, 0, 0, 1, 0, 0, 1) + struct.pack("<Qf", 10, prob) +
                  struct.pack("<QIQI", 1, 10, 20, 2) + struct.pack("<QQ", 0, 0))
    if ok:
        assert lt.checkpoint_info(f)["num_walkers"] == 10
    else:
        with pytest.raises(lt.LTError, match="LT_ERR_FORMAT.*stop probability"):
            lt.checkpoint_info(f)


@pytest.mark.gpu
@pytest.mark.parametrize("prob", SMALL)
def test_refused_calls(lt, require_gpu, prob):
    V = 1000
    rp, col = 4 * np.arange(V + 1, dtype=np.uint64), np.arange(4 * V, dtype=np.uint32) % V
    resident = lt.Engine(lt.Graph.from_csr(rp, col, 1 << 20))
    ooc = lt.Engine(lt.Graph.from_csr(rp, col, 1 << 10), partitions=12, sched=4)
    for call in (lambda: resident.ppr(0, 10, prob), lambda: ooc.ppr(0, 10, prob),
                 lambda: resident.ppr_batch([0], [10], [1], prob), lambda: lt.Server(ooc, prob=prob)):
        with pytest.raises(lt.LTError, match="LT_ERR_INVALID.*stop probability"):
            call()
