"""Host arrays at addresses that are no multiple of 8 (views into packed
records or byte buffers): the same results as from aligned ones, through every
call that reads or writes a caller's array."""
import ctypes

import numpy as np
import pytest

from hadronic_afterburner_toolkit_gb300 import bf, engine, synth

pytestmark = pytest.mark.gpu
_PD = ctypes.POINTER(ctypes.c_double)
P = dict(qnpts=11, q_min=-0.15, q_max=0.15, n_KT=5, KT_min=0.0, KT_max=1.0, n_Kphi=4,
         azimuthal_flag=0, invariant_radius_flag=1, long_comoving_boost=1,
         needed_number_of_pairs=1e18)


def at_offset(a, offset):
    raw = np.zeros(8 * a.size + 16, np.uint8)
    start = -raw.ctypes.data % 8 + offset
    v = raw[start:start + 8 * a.size].view(np.float64)
    v[:] = a
    assert v.ctypes.data % 8 == offset and v.flags.c_contiguous
    return v


def columns():
    ev = synth.generate(4, 90.0, seed=5, sigma_xy=3.0, tau_mean=4.0)
    return [np.ascontiguousarray(getattr(ev, k)) for k in
            ("px", "py", "pz", "E", "x", "y", "z", "t")]


@pytest.mark.parametrize("offset", [1, 4])
def test_binning_and_reading(offset):
    c = columns()
    # all columns off, one column off
    variants = [c, [at_offset(a, offset) for a in c],
                [at_offset(a, offset) if k == 3 else a for k, a in enumerate(c)]]
    got = []
    for v in variants:
        eng = engine.Engine(**P)
        eng.bin_same(v)
        eng.bin_mixed(v[:4], [a[:100] for a in v[:4]])
        eng.bin_batch([("same", v), ("mixed", v[:4], [a[50:] for a in v[:4]])])
        got.append(eng.hist())
        if v is variants[1]:  # read into such arrays
            n, nq = int(eng.L.hbt_n_bins(eng.handle)), P["n_KT"] * P["qnpts"]
            out = [at_offset(np.zeros(n), offset) for _ in range(6)]
            qi = [at_offset(np.zeros(nq), offset) for _ in range(4)]
            assert eng.L.hbt_read_hist(eng.handle, *[a.ctypes.data_as(_PD) for a in out]) == 0
            assert eng.L.hbt_read_qinv(eng.handle, *[a.ctypes.data_as(_PD) for a in qi]) == 0
            for a, k in zip(out + qi, ("count", "q_out", "q_side", "q_long", "num", "den",
                                       "qinv_sum", "qinv_num", "qinv_count", "qinv_den")):
                assert np.array_equal(a, got[-1][k]), k
        eng.close()
    assert got[0]["count"].sum() > 100 and got[0]["den"].sum() > 100
    for h in got[1:]:
        for k in ("count", "den", "qinv_count", "qinv_den"):
            assert np.array_equal(h[k], got[0][k]), k
        # sums of values up to 1 in another order
        for k in ("num", "q_out", "qinv_sum"):
            n = np.maximum(got[0]["qinv_count" if k == "qinv_sum" else "count"], 1.0)
            assert np.all(np.abs(h[k] - got[0][k]) <= 2.0 ** -52 * n * n), k


@pytest.mark.parametrize("offset", [1, 4])
def test_balance_function(offset):
    rng = np.random.default_rng(3)
    off = np.arange(0, 501, 100)
    phi, y = rng.uniform(-3.0, 3.0, 500), rng.normal(0.0, 1.0, 500)
    jobs = [(0, 0, e, 0, f, 0, 0.0) for e in range(5) for f in range(5)]
    got = []
    for lists in ([(off, phi, y)], [(off, at_offset(phi, offset), at_offset(y, offset))],
                  [(off, phi, at_offset(y, offset))]):
        b = bf.BfEngine(21, 2.0)
        b.bin(lists, jobs)
        got.append(b.hist(0))
        out = at_offset(np.zeros(21 * bf.NPHI), offset)
        assert b.L.hbt_bf_read(b._h, 0, out.ctypes.data_as(_PD)) == 0
        assert np.array_equal(out.reshape(21, bf.NPHI), got[-1])
        b.close()
    assert got[0].sum() > 1000
    assert np.array_equal(got[1], got[0]) and np.array_equal(got[2], got[0])
