"""The fixed-point pair values (csrc/hbt_fixed.cuh) at the edges of their
range: positions and energies on both sides of the limits (634 fm, 8 GeV),
momenta and positions of every size, beside particles well inside; against
the oracle.  Tolerance: both sides round four products of a momentum and a
position difference and their sum at 2^-53, so a pair's phase differs by at
most 16 2^-53 (2 p_max) (2 x_max) / hbarC, and its cosine by no more."""
import numpy as np
import pytest

import oracle_lib
from hadronic_afterburner_toolkit_gb300 import engine

pytestmark = pytest.mark.gpu
LIMIT_FM = 2.0 ** 18 * 2.0 * np.pi * 0.197327053 / 512.0


def particles(n, seed, x_scale, p_scale):
    rng = np.random.default_rng(seed)
    px, py = rng.normal(0.0, 0.1, n), rng.normal(0.0, 0.1, n)
    pz = rng.normal(0.0, 0.05, n)
    px[: n // 2] += p_scale      # half of them close together at a high momentum
    px[::9] = rng.choice([1e-9, -3e-5, 0.0625, 0.25, -0.5], px[::9].size)
    E = np.sqrt(0.13957 ** 2 + px * px + py * py + pz * pz)
    pos = [x_scale * rng.normal(0.0, 1.0, n) for _ in range(4)]
    edge = LIMIT_FM * np.array([1.0 - 1e-12, 1.0, 1.0 + 1e-12, -1.0, 0.5, 1e-12])
    for k, c in enumerate(pos):
        c[k::7] = rng.choice(edge, c[k::7].size)
    return [px, py, pz, E] + pos


@pytest.mark.parametrize("precision", [engine.PRECISION_FP64, engine.PRECISION_DF64,
                                       engine.PRECISION_FP32W])
@pytest.mark.parametrize("boost", [0, 1])
@pytest.mark.parametrize("x_scale,p_scale", [(3.0, 0.0), (3.0, 7.9), (300.0, 0.4), (5000.0, 8.0)])
def test_values_equal_the_oracle(x_scale, p_scale, boost, precision):
    p = dict(qnpts=9, q_min=-0.2, q_max=0.2, n_KT=4, KT_min=0.0, KT_max=12.0, n_Kphi=4,
             azimuthal_flag=0, invariant_radius_flag=0, long_comoving_boost=boost,
             needed_number_of_pairs=1e18)
    cols = particles(300, 5, x_scale, p_scale)
    eng, orc = engine.Engine(precision=precision, **p), oracle_lib.Oracle(**p)
    for x in (eng, orc):
        x.bin_same(cols)
    h, o = eng.hist(), orc.hist()
    eng.close()
    assert np.array_equal(h["count"], o["count"]) and o["count"].sum() > 1000
    x_max = max(np.abs(c).max() for c in cols[4:])
    phase = 16 * 2.0 ** -53 * 2 * cols[3].max() * 2 * x_max / 0.197327053
    if precision == engine.PRECISION_DF64:
        phase *= 64.0  # its stated accuracy allows 48-bit values
    n = np.maximum(o["count"], 1.0)
    # FP32 weights: the form's stated bound
    fp32 = precision == engine.PRECISION_FP32W
    assert np.all(np.abs(h["num"] - o["num"]) <= n * ((1e-5 if fp32 else 1e-15) + phase))
    for k in ("q_out", "q_side", "q_long"):
        assert np.all(np.abs(h[k] - o[k]) <= (1e-5 if fp32 else 1e-12) * 0.225 * n), k
