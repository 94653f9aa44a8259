"""Particles at rapidities up to and past the limits of the screen's light-cone
terms (9.7) and of the cull's boxes (10.7): counts equal to the oracle's, and
tile pairs far apart in rapidity culled."""
import numpy as np
import pytest

import oracle_lib
from hadronic_afterburner_toolkit_gb300 import engine

pytestmark = pytest.mark.gpu


def particles(n, seed, lo, hi, m=0.13957):
    rng = np.random.default_rng(seed)
    pt, ph = rng.exponential(0.15, n), rng.uniform(0.0, 2.0 * np.pi, n)
    y = rng.uniform(lo, hi, n) * rng.choice([-1.0, 1.0], n)
    y[1::3] = y[::3][: y[1::3].size] + rng.choice([0.0, 1e-2, 0.3], y[1::3].size)  # neighbours
    px, py = pt * np.cos(ph), pt * np.sin(ph)
    mt = np.sqrt(m ** 2 + pt * pt)
    cols = [px, py, mt * np.sinh(y), mt * np.cosh(y)]
    return cols + [rng.normal(0.0, 5.0, n) for _ in range(4)]


@pytest.mark.parametrize("precision", [engine.PRECISION_FP64, engine.PRECISION_FP32W])
@pytest.mark.parametrize("boost,qinv,n_kphi", [(1, 0, 0), (1, 1, 3), (0, 0, 3), (0, 1, 0)])
@pytest.mark.parametrize("lo,hi", [(0.0, 8.5), (8.0, 8.6), (9.5, 9.9), (7.5, 12.0)])
def test_counts_equal_the_oracle(lo, hi, boost, qinv, n_kphi, precision):
    p = dict(qnpts=21, q_min=-0.2, q_max=0.2, n_KT=5, KT_min=0.0, KT_max=1.0,
             n_Kphi=n_kphi or 4, azimuthal_flag=int(n_kphi > 0), invariant_radius_flag=qinv,
             long_comoving_boost=boost, needed_number_of_pairs=1e18)
    a, b = particles(700, 3, lo, hi), particles(300, 4, lo, hi)
    eng, orc = engine.Engine(precision=precision, **p), oracle_lib.Oracle(**p)
    for x in (eng, orc):
        x.bin_same(a)
        x.bin_mixed(a[:4], b[:4])
    h, o = eng.hist(), orc.hist()
    eng.close()
    for k in ("count", "den", "qinv_count", "qinv_den", "ctr_num", "ctr_den"):
        assert np.array_equal(np.asarray(h[k]), np.asarray(o[k])), k


def test_tiles_far_apart_in_rapidity_are_culled():
    """Two halves 14 units apart: of 32 tiles' 528 pairs the 256 between the
    halves can bin nothing, but for those of a tile with both."""
    a = particles(4096, 5, 7.0, 8.5)
    eng = engine.Engine(long_comoving_boost=1)
    eng.bin_same(a)
    s = eng.stats()
    eng.close()
    assert s["tiles_same"] == 528
    assert s["tiles_same_kept"] <= 528 - 256 + 32
