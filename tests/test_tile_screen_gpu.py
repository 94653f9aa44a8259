"""The tile screen (csrc/hbt_screen.cuh) at the edges of its range: list
sizes around the 128-particle tile and its two-particle steps, small and even
q grids, rapidities past the light-cone terms' limit, pairs whose K_perp is
lost to cancellation, equal particles; against the oracle, counts equal."""
import numpy as np
import pytest

import oracle_lib
from hadronic_afterburner_toolkit_gb300 import engine

pytestmark = pytest.mark.gpu


def particles(n, seed, y_max):
    rng = np.random.default_rng(seed)
    pt, ph = rng.exponential(0.2, n), rng.uniform(0.0, 2.0 * np.pi, n)
    y = rng.uniform(-y_max, y_max, n)
    px, py = pt * np.cos(ph), pt * np.sin(ph)
    for k in range(1, n, 5):  # nearby, equal and opposite particles
        px[k], py[k], y[k] = px[k - 1], py[k - 1], y[k - 1] + rng.choice([0.0, 1e-3, 0.2])
        if k % 10 == 1:
            px[k], py[k] = -px[k] * (1.0 + 1e-9), -py[k]
    mt = np.sqrt(0.13957 ** 2 + px * px + py * py)
    cols = [px, py, mt * np.sinh(y), mt * np.cosh(y)]
    return cols + [rng.normal(0.0, 5.0, n) for _ in range(4)]


@pytest.mark.parametrize("qnpts,q_min,q_max", [(2, -0.15, 0.15), (40, -0.15, 0.15),
                                               (41, -0.1, 0.3)])
@pytest.mark.parametrize("boost,n_kphi,psi,y_max", [(1, 0, 0.0, 1.0), (1, 5, 2.9, 8.0),
                                                    (0, 3, -0.4, 1.5)])
@pytest.mark.parametrize("n", [2, 3, 127, 128, 129, 383])
def test_counts_equal_the_oracle(n, boost, n_kphi, psi, y_max, qnpts, q_min, q_max):
    p = dict(qnpts=qnpts, q_min=q_min, q_max=q_max, n_KT=5, KT_min=0.05, KT_max=0.9,
             n_Kphi=n_kphi or 4, azimuthal_flag=int(n_kphi > 0), invariant_radius_flag=0,
             long_comoving_boost=boost, needed_number_of_pairs=1e18)
    a, b = particles(n, 11 * n + boost, y_max), particles(n + 64, 7 * n + 1, y_max)
    eng, orc = engine.Engine(**p), oracle_lib.Oracle(**p)
    for x in (eng, orc):
        x.set_psi_ref(psi)
        x.bin_same(a)
        x.bin_mixed(a[:4], b[:4])
    h, o = eng.hist(), orc.hist()
    eng.close()
    for k in ("count", "den", "ctr_num", "ctr_den"):
        assert np.array_equal(np.asarray(h[k]), np.asarray(o[k])), k
    # the phase's rounding grows with the energies: four terms of at most
    # 2 E_max 60 fm / hbarC, each rounded at 2^-53
    e_max = 1.0 + max(a[3].max(), b[3].max())
    for k, scale in (("num", e_max), ("q_out", max(abs(q_min), q_max))):
        assert np.all(np.abs(h[k] - o[k]) <= 1e-12 * np.maximum(o["count"], 1.0) * scale), k
