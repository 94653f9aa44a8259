"""The q_inv part of the tile screen (csrc/hbt_screen.cuh screen_qinv) where it
can go wrong: pairs whose q_inv^2 is within its rounding of zero on either side
(particles of different masses, momenta of a few digits), on grids with and
without a bin centred at zero; rapidities past the light-cone terms' limit,
pairs whose K_perp is lost to cancellation, equal particles, list sizes around
the 128-particle tile; against the oracle, counts equal."""
import numpy as np
import pytest

import oracle_lib
from hadronic_afterburner_toolkit_gb300 import engine

pytestmark = pytest.mark.gpu
FORMS = [engine.PRECISION_FP64, engine.PRECISION_DF64, engine.PRECISION_FP32W]


def both(p, precision, a, b):
    eng, orc = engine.Engine(precision=precision, **p), oracle_lib.Oracle(**p)
    for x in (eng, orc):
        x.bin_same(a)
        x.bin_mixed(a[:4], b[:4])
    h, o = eng.hist(), orc.hist()
    eng.close()
    for k in ("count", "den", "qinv_count", "qinv_den", "ctr_num", "ctr_den", "ctr_num_qinv",
              "ctr_den_qinv"):
        assert np.array_equal(np.asarray(h[k]), np.asarray(o[k])), k
    # each value lies in the window; the sums' own rounding
    tol = 1e-12 * max(abs(p["q_min"]), p["q_max"]) * np.maximum(o["qinv_count"], 1.0)
    assert np.all(np.abs(h["qinv_sum"] - o["qinv_sum"]) <= tol)
    return o


def zero_pairs(seed):
    """Pairs whose energy difference is their momentum difference's length to
    1e-9 .. 1e-5, and one of 6-digit momenta."""
    rng = np.random.default_rng(seed)
    rows = [[0.959364, -0.650772, -0.244581, 1.192972], [0.959387, -0.650786, -0.244583, 1.192999]]
    for _ in range(150):
        p = rng.normal(0.0, 0.3, 3)
        E = np.sqrt(0.13957 ** 2 + p @ p)
        d = rng.normal(0.0, 1.0, 3) * 10.0 ** rng.uniform(-5.0, -3.0)
        dE = np.linalg.norm(d) * (1.0 + rng.choice([-1, 1]) * 10.0 ** rng.uniform(-9.0, -5.0))
        rows += [[*p, E], [*(p + d), E + dE]]
    m = np.array(rows).T
    return [np.ascontiguousarray(c) for c in m] + [rng.normal(0.0, 4.0, m.shape[1]) for _ in range(4)]


@pytest.mark.parametrize("precision", FORMS)
@pytest.mark.parametrize("boost", [0, 1])
@pytest.mark.parametrize("qnpts,q_min,q_max", [(41, -0.15, 0.15), (40, -0.15, 0.15),
                                               (3, -0.2, 0.2), (21, 0.0, 0.3)])
def test_sign_of_q_inv_squared(qnpts, q_min, q_max, boost, precision):
    p = dict(qnpts=qnpts, q_min=q_min, q_max=q_max, n_KT=5, KT_min=0.0, KT_max=2.0, n_Kphi=4,
             azimuthal_flag=0, invariant_radius_flag=1, long_comoving_boost=boost,
             needed_number_of_pairs=1e18)
    a = zero_pairs(3)
    o = both(p, precision, a, a)
    assert o["qinv_count"].sum() > 100


def edge_particles(n, seed, y_max):
    rng = np.random.default_rng(seed)
    pt, ph = rng.exponential(0.2, n), rng.uniform(0.0, 2.0 * np.pi, n)
    y = rng.uniform(-y_max, y_max, n)
    m = rng.choice([0.13957, 0.49368], n)
    px, py = pt * np.cos(ph), pt * np.sin(ph)
    for k in range(1, n, 5):  # nearby, equal and opposite particles
        px[k], py[k], y[k] = px[k - 1], py[k - 1], y[k - 1] + rng.choice([0.0, 1e-3, 0.2])
        if k % 10 == 1:
            px[k], py[k] = -px[k] * (1.0 + 1e-9), -py[k]
    mt = np.sqrt(m ** 2 + px * px + py * py)
    cols = [px, py, mt * np.sinh(y), mt * np.cosh(y)]
    return cols + [rng.normal(0.0, 5.0, n) for _ in range(4)]


@pytest.mark.parametrize("precision", [engine.PRECISION_FP64, engine.PRECISION_FP32W])
@pytest.mark.parametrize("boost,n_kphi,y_max", [(1, 0, 1.0), (1, 5, 8.0), (0, 3, 1.5),
                                                (0, 0, 8.0)])
@pytest.mark.parametrize("n", [2, 127, 129, 383])
def test_edges_equal_the_oracle(n, boost, n_kphi, y_max, precision):
    p = dict(qnpts=41, q_min=-0.15, q_max=0.15, n_KT=5, KT_min=0.05, KT_max=0.9,
             n_Kphi=n_kphi or 4, azimuthal_flag=int(n_kphi > 0), invariant_radius_flag=1,
             long_comoving_boost=boost, needed_number_of_pairs=1e18)
    both(p, precision, edge_particles(n, 11 * n + boost, y_max),
         edge_particles(n + 64, 7 * n + 1, y_max))


@pytest.mark.parametrize("precision", FORMS)
@pytest.mark.parametrize("boost", [0, 1])
def test_values_are_the_reference_expressions(boost, precision):
    """Few pairs to a bin: each q_inv is the FP64 expression's value, so that a
    bin's sum differs by the order of its additions only, n - 1 roundings of
    the sum each way."""
    p = dict(qnpts=41, q_min=-0.15, q_max=0.15, n_KT=5, KT_min=0.0, KT_max=2.0, n_Kphi=4,
             azimuthal_flag=0, invariant_radius_flag=1, long_comoving_boost=boost,
             needed_number_of_pairs=1e18)
    for seed in range(4):
        a = edge_particles(90, 100 + seed, 1.0)
        eng, orc = engine.Engine(precision=precision, **p), oracle_lib.Oracle(**p)
        for x in (eng, orc):
            x.bin_same(a)
        h, o = eng.hist(), orc.hist()
        eng.close()
        assert np.array_equal(h["qinv_count"], o["qinv_count"]) and o["qinv_count"].sum() > 100
        tol = 2.0 ** -52 * np.maximum(o["qinv_count"] - 1.0, 0.0) * o["qinv_sum"]
        assert np.all(np.abs(h["qinv_sum"] - o["qinv_sum"]) <= tol)
