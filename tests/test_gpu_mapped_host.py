"""Which host memory the kernels write results to themselves (the library's mapped_host): only a range inside one page-locked
allocation or registered region; everything else takes a copy."""
import ctypes
import mmap

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mapped(lt, require_gpu):
    f = lt.lib["_ZN2lt11mapped_hostEPKvm"]  # lt::mapped_host(void const *, unsigned long)
    f.argtypes, f.restype = [ctypes.c_void_p, ctypes.c_size_t], ctypes.c_void_p
    return f


def test_one_allocation(lt, mapped):
    a = lt.pinned_empty(1000003, np.uint8)
    p = a.ctypes.data
    for at, n in ((0, 1000003), (0, 1), (8, 1000), (1000002, 1), (17, 0)):
        assert mapped(p + at, n) == p + at  # unified addressing
    for at, n in ((0, 1000004), (1000002, 2), (1000003, 1), (8, 1 << 63), (8, 2**64 - 1)):
        assert mapped(p + at, n) is None
    plain = np.zeros(1000, np.uint8)
    assert mapped(plain.ctypes.data, 8) is None and mapped(None, 8) is None


def test_registered_regions(lt, mapped):
    """Two registered regions with pageable memory between them, and one that touches the first."""
    import torch
    rt = torch.cuda.cudart()
    m = mmap.mmap(-1, 4 << 20)
    p = ctypes.addressof(ctypes.c_char.from_buffer(m))
    regions = [(p, 1 << 20), (p + (3 << 20), 1 << 20), (p + (1 << 20), 4096)]
    done = []
    try:
        for at, n in regions:
            assert int(rt.cudaHostRegister(at, n, 0)) == 0
            done.append(at)
        for at, n in regions:
            assert mapped(at, n) == at and mapped(at + 100, n - 100) == at + 100
            assert mapped(at, n + 1) is None
        assert mapped(p, 4 << 20) is None and mapped(p + 4096, (4 << 20) - 8192) is None
        assert mapped(p + (2 << 20), 8) is None
    finally:
        for at in done:
            rt.cudaHostUnregister(at)


def test_device_memory(lt, mapped):
    import torch
    t = torch.zeros(1000, dtype=torch.int64, device="cuda")
    assert mapped(t.data_ptr(), 8000) is None
