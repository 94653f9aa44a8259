"""Pairs of particles outside the fixed-point columns' range (positions past
634 fm, energies past 8 GeV), which are collected and summed 32 at a time
(csrc/hbt_tile.cuh far_values): none, few, half or all of a list, through the
batched and grid kernels and under a binding cap; against the oracle.
Tolerances as in tests/test_fixed_values_gpu.py: both sides round four products
of a momentum and a position difference and their sum at 2^-53."""
import numpy as np
import pytest

import oracle_lib
from hadronic_afterburner_toolkit_gb300 import engine

pytestmark = pytest.mark.gpu


def particles(n, seed, share, far_energy):
    rng = np.random.default_rng(seed)
    px, py, pz = rng.normal(0.0, 0.15, (3, n))
    pos = rng.normal(0.0, 6.0, (4, n))
    far = rng.random(n) < share
    if far_energy:
        pz[far] += 9.0
    else:
        pos[:, far] *= 400.0
    E = np.sqrt(0.13957 ** 2 + px * px + py * py + pz * pz)
    return [np.ascontiguousarray(c) for c in (px, py, pz, E, *pos)]


@pytest.mark.parametrize("kernel,cap,n_kphi,qinv", [(0, 1e18, 0, 0), (0, 1e18, 3, 1),
                                                    (2, 1e18, 3, 0), (0, 2e3, 0, 0)])
@pytest.mark.parametrize("boost", [0, 1])
@pytest.mark.parametrize("share", [0.02, 0.5, 1.0])
@pytest.mark.parametrize("far_energy", [False, True])
def test_sums_equal_the_oracle(far_energy, share, boost, kernel, cap, n_kphi, qinv):
    p = dict(qnpts=11, q_min=-0.2, q_max=0.2, n_KT=4, KT_min=0.0, KT_max=1.0,
             n_Kphi=n_kphi or 4, azimuthal_flag=int(n_kphi > 0), invariant_radius_flag=qinv,
             long_comoving_boost=boost, needed_number_of_pairs=cap)
    cols = particles(500, 7, share, far_energy)
    eng, orc = engine.Engine(kernel=kernel, **p), oracle_lib.Oracle(**p)
    for x in (eng, orc):
        x.bin_same(cols)
    h, o = eng.hist(), orc.hist()
    eng.close()
    for k in ("count", "qinv_count", "ctr_num"):
        assert np.array_equal(np.asarray(h[k]), np.asarray(o[k])), k
    assert o["count"].sum() > 1000
    x_max = max(np.abs(c).max() for c in cols[4:])
    phase = 16 * 2.0 ** -53 * 2 * cols[3].max() * 2 * x_max / 0.197327053
    for k, c in (("num", "count"), ("qinv_num", "qinv_count")):
        n = np.maximum(o[c], 1.0)
        assert np.all(np.abs(h[k] - o[k]) <= n * (1e-15 + phase)), k
    n = np.maximum(o["count"], 1.0)
    for k in ("q_out", "q_side", "q_long"):
        assert np.all(np.abs(h[k] - o[k]) <= 1e-12 * 0.225 * n), k
