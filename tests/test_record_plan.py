"""The memory that the candidate records of the FP32 sphere list build take: a stated
budget is kept but for the smallest plan, which every build had before."""
import ctypes as C

import pytest


def _plan(lib, n, mesh, budget):
    out = (C.c_uint32 * 2)()
    assert lib.dem_selftest_record_plan(n, mesh, budget, out) == 0
    return tuple(out)


@pytest.mark.parametrize("n", [1, 7, 1000, 2_000_000, 1 << 24, 170_000_000, (1 << 31) - 1])
def test_plan(native_lib, n):
    small, plain, full = 64 * n, 256 * n, 1024 * n
    assert _plan(native_lib, n, 0, plain) == (16, 0) == _plan(native_lib, n, 0, full)
    assert _plan(native_lib, n, 0, plain - 1) == (4, 0) == _plan(native_lib, n, 0, small) == _plan(native_lib, n, 0, 1)
    assert _plan(native_lib, n, 1, full) == (16, 48)
    assert _plan(native_lib, n, 1, full - 1) == (16, 0) == _plan(native_lib, n, 1, plain)
    assert _plan(native_lib, n, 1, plain - 1) == (4, 0)
