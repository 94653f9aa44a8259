"""The double-float form runs the FP64 form's kernels: equal counts, and sums
that differ by the order of their additions only (n - 1 roundings each way of
sums of at most n times the largest value)."""
import numpy as np
import pytest

from hadronic_afterburner_toolkit_gb300 import engine
from test_far_particles_gpu import particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("qinv", [0, 1])
@pytest.mark.parametrize("boost", [0, 1])
@pytest.mark.parametrize("share", [0.0, 0.3])
def test_sums_equal_the_fp64_form(share, boost, qinv):
    p = dict(qnpts=11, q_min=-0.2, q_max=0.2, n_KT=4, KT_min=0.0, KT_max=1.0, n_Kphi=4,
             azimuthal_flag=0, invariant_radius_flag=qinv, long_comoving_boost=boost,
             needed_number_of_pairs=1e18)
    cols = particles(600, 9, share, False)
    h = []
    for form in (engine.PRECISION_FP64, engine.PRECISION_DF64):
        eng = engine.Engine(precision=form, **p)
        eng.bin_same(cols)
        h.append(eng.hist())
        eng.close()
    a, b = h
    assert a["count"].sum() > 1000
    for k in ("count", "qinv_count"):
        assert np.array_equal(a[k], b[k]), k
    for k, c, top in (("num", "count", 1.0), ("q_out", "count", 0.22), ("q_side", "count", 0.22),
                      ("q_long", "count", 0.22), ("qinv_sum", "qinv_count", 0.22),
                      ("qinv_num", "qinv_count", 1.0)):
        n = a[c]
        assert np.all(np.abs(a[k] - b[k]) <= 2.0 ** -52 * n * np.maximum(n - 1.0, 0.0) * top), k
