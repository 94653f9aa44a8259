"""Which way the library reads or writes a caller's host array
(csrc/hbt_hostmem.h), without a device."""
import ctypes

import numpy as np
import pytest

from hadronic_afterburner_toolkit_gb300 import build, engine

KERNEL, COPIES = 2, 1


@pytest.fixture(scope="module")
def route():
    build.build_gpu()
    fn = engine.load().hbt_check_host_route
    fn.restype, fn.argtypes = ctypes.c_int32, [ctypes.c_void_p]
    return fn


@pytest.mark.parametrize("offset", range(9))
def test_kernels_take_aligned_arrays_only(route, offset):
    raw = np.zeros(64 + 9, np.uint8)
    start = -raw.ctypes.data % 8 + offset
    a = raw[start:start + 32].view(np.float64)
    # what the binding passes on: it leaves the address as it is
    p = engine._arr(a).ctypes.data
    assert p == a.ctypes.data
    assert route(p) == (KERNEL if offset % 8 == 0 else COPIES)
