"""The pair kernels' cosine of fixed-point phases (csrc/hbt_fixed.cuh cos_fixed)
with the kernels' table, against the host's extended-precision cosine: within
its stated 4e-16 over the period, at the 2048 table points, half way between
them, one unit either side of those, and at phases of 2^25 periods."""
import ctypes

import numpy as np
import pytest

from hadronic_afterburner_toolkit_gb300 import engine

pytestmark = pytest.mark.gpu
PERIOD = 1 << 46  # in 2^-37 steps of 2 pi / 512


def device(steps):
    L = engine.load()
    fn = L.hbt_check_cos_fixed
    fn.restype = ctypes.c_int32
    fn.argtypes = [ctypes.c_int, ctypes.c_int64, ctypes.c_void_p, ctypes.c_void_p]
    steps = np.ascontiguousarray(steps, dtype=np.int64)
    out = np.empty(len(steps))
    assert fn(0, len(steps), steps.ctypes.data, out.ctypes.data) == 0
    return out


def want(steps):
    # within an eighth of a period of the axes, where the angle is small
    x = steps[:, 0] % PERIOD
    quad = ((x + PERIOD // 8) // (PERIOD // 4)) % 4
    rest = (x + PERIOD // 8) % (PERIOD // 4) - PERIOD // 8
    t = rest.astype(np.longdouble) + steps[:, 1].astype(np.longdouble) * np.longdouble(2.0) ** -30
    t = t * (np.longdouble("3.14159265358979323846264338327950288") / (PERIOD // 2))
    c, s = np.cos(t), np.sin(t)
    return np.choose(quad, [c, -s, -c, s])


def test_cos_fixed():
    rng = np.random.default_rng(1)
    cell = PERIOD // 2048
    points = np.arange(-3000, 3000, dtype=np.int64) * cell
    hh = np.concatenate([rng.integers(-PERIOD, PERIOD, 300000), points, points + cell // 2,
                         points + cell // 2 - 1, points + cell // 2 + 1, points - 1, points + 1,
                         rng.integers(-(1 << 62) + 1, (1 << 62) - 1, 300000)])
    hl = rng.integers(0, 1 << 30, hh.size)
    edge = rng.random(hh.size) < 0.2
    hl[edge] = rng.choice([0, 1, (1 << 30) - 1], edge.sum())
    steps = np.stack([hh, hl], axis=1)
    assert np.max(np.abs(device(steps).astype(np.longdouble) - want(steps))) < 4e-16
