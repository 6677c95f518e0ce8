"""Which arrays the copy kernel of dem_set_particles and dem_get_particles takes: those
that lie inside an allocation of the device.  One that is shorter than the particles is
left to cudaMemcpyAsync, which refuses it."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [8, 4096, 1 << 20, (1 << 21) + 24])
def test_only_whole_ranges(native_lib, size):
    import torch

    torch.zeros(1, device="cuda")  # the device's context
    drv = C.CDLL("libcuda.so.1")
    p = C.c_uint64()
    assert drv.cuMemAlloc_v2(C.byref(p), C.c_size_t(size)) == 0
    inside = C.c_int(-1)

    def ask(at, nbytes):
        assert native_lib.dem_selftest_copy_range(C.c_void_p(at), nbytes, C.byref(inside)) == 0
        return inside.value

    try:
        assert ask(p.value, size) == 1 and ask(p.value + size - 1, 1) == 1 and ask(p.value + size // 2, size // 2) == 1
        for at, nbytes in ((p.value, size + 1), (p.value + 1, size), (p.value + size // 2, size), (p.value, 1 << 40),
                           (p.value + size - 1, 2), (p.value + 1, (1 << 64) - 1)):
            assert ask(at, nbytes) == 0
        host = np.zeros(size, np.uint8)
        assert ask(host.ctypes.data, 1) == 0
        pinned = torch.zeros(size, dtype=torch.uint8, pin_memory=True)
        assert ask(pinned.data_ptr(), 1) == 0
        t = torch.zeros(size, dtype=torch.uint8, device="cuda")
        assert ask(t.data_ptr(), size) == 1
    finally:
        drv.cuMemFree_v2(p)
