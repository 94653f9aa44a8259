"""Batched binning where its preparation and its launches change course: list
lengths at the edges of the ordering blocks (1024, 2048, 4096 and 8192 rows)
and of the device sort beyond them, and numbers of tile pairs for which a tile
pair is split into 16 parts down to one.  Counts must be the oracle's; the sums
agree to the tolerance of tests/parity.py."""
import numpy as np
import pytest

import oracle_lib
import parity

pytestmark = pytest.mark.gpu

P = dict(qnpts=9, q_min=-0.12, q_max=0.12, n_KT=4, KT_min=0.0, KT_max=1.0, n_Kphi=4,
         azimuthal_flag=0, invariant_radius_flag=0, needed_number_of_pairs=1e18)


def _cols(n, seed):
    rng = np.random.default_rng(seed)
    px, py, pz = rng.normal(0.0, 0.3, (3, n))
    e = np.sqrt(px * px + py * py + pz * pz + 0.13957 ** 2)
    return [px, py, pz, e] + list(rng.normal(0.0, 4.0, (4, n)))


@pytest.mark.parametrize("boost", [0, 1])
@pytest.mark.parametrize("n", [100, 700, 1024, 1025, 2048, 2049, 4096, 4097, 8192, 8193])
def test_list_lengths_and_parts(n, boost):
    from hadronic_afterburner_toolkit_gb300 import engine
    p = dict(P, long_comoving_boost=boost)
    eng, orc = engine.Engine(**p), oracle_lib.Oracle(**p)
    c, l1, l2 = _cols(n, n), _cols(200, n + 1)[:4], _cols(n, n + 2)[:4]
    for o in (eng, orc):
        o.set_psi_ref(0.0)
        o.bin_same(c)
        o.bin_mixed(l1, l2)
    h = orc.hist()
    assert h["count"].sum() > 0 and h["den"].sum() > 0
    parity.compare(eng.hist(), h, 0.2)
