"""The cut row of a binding cap on the GPU, at the edges of the column chunks
(256 columns to a block) its pairs are admitted in.

Which pairs are admitted is exact, so the counts must equal the oracle's; the
sums agree to the tolerance of tests/parity.py."""
import numpy as np
import pytest

import oracle_lib
import parity

pytestmark = pytest.mark.gpu

P = dict(qnpts=7, q_min=-0.15, q_max=0.15, n_KT=2, KT_min=0.0, KT_max=1.0, n_Kphi=4,
         azimuthal_flag=0, invariant_radius_flag=0, long_comoving_boost=1)


def _cols(n, seed):
    rng = np.random.default_rng(seed)
    px, py, pz = rng.normal(0.0, 0.08, (3, n))
    e = np.sqrt(px * px + py * py + pz * pz + 0.13957 ** 2)
    return [px, py, pz, e] + list(rng.normal(0.0, 4.0, (4, n)))


@pytest.mark.parametrize("qinv", [0, 1])
@pytest.mark.parametrize("n", [2, 256, 257, 513, 770])
@pytest.mark.parametrize("cap", [1, 40, 260])
def test_cut_row_across_column_chunks(cap, n, qinv):
    from hadronic_afterburner_toolkit_gb300 import engine
    p = dict(P, needed_number_of_pairs=cap, invariant_radius_flag=qinv)
    eng, orc = engine.Engine(**p), oracle_lib.Oracle(**p)
    c, l1, l2 = _cols(n, n), _cols(3, n + 1)[:4], _cols(n, n + 2)[:4]
    for o in (eng, orc):
        o.set_psi_ref(0.0)
        o.bin_same(c)
        o.bin_mixed(l1, l2)
    h = orc.hist()
    if n > 2 and cap < 260:
        assert (h["ctr_num"] == cap + 1).any() and (h["ctr_den"] == cap + 1).any()
    parity.compare(eng.hist(), h, 0.2)
