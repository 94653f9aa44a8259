"""Balance-function binning on the GPU where its loop changes course: list
sizes at the edges of the groups of 4 pairs, the 128-particle tiles and the 256
staged particles, a list against itself (every particle with itself is
skipped), rotations of several magnitudes, rapidities far outside the window,
and a rapidity that is not a number.  Counts must be the oracle's."""
import numpy as np
import pytest

import oracle_lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("na,nb", [(1, 1), (3, 5), (127, 255), (128, 256), (129, 257), (260, 513)])
def test_bf_group_and_stage_edges(na, nb):
    from hadronic_afterburner_toolkit_gb300 import bf
    rng = np.random.default_rng(na)
    lists = []
    for n in (na, nb):
        y, phi = rng.normal(0.0, 0.7, n), rng.uniform(-np.pi, np.pi, n)
        if n > 2:
            y[1], phi[2] = 3.0e5, 9.0e4
        if n > 4:
            y[4] = np.nan
        lists.append((np.array([0, n], np.int64), phi, y))
    jobs = [(0, 0, 0, 1, 0, 0, 0.0), (1, 1, 0, 1, 0, 0, 0.0)]
    jobs += [(2 + r, 0, 0, 1, 0, 1, rot) for r, rot in enumerate([0.0, 6.28, -50.0, 1.0e5, 3.0e7])]
    eng = bf.BfEngine(21, 1.5)
    eng.bin(lists, bf.job_array(jobs))
    orc = oracle_lib.BfOracle(particle_alpha=1, particle_beta=2, BpT_min=-1.0, BpT_max=10.0,
                              Bnpts=21, Brap_max=1.5, rap_type=1, seed=1)
    L = oracle_lib._bf_lib()
    for (h, la, _, lb, _, mx, rot) in jobs:
        # converting a NaN quotient to an integer is undefined in the reference
        # (x86 and the GPU leave the histogram, Arm gives row 0): the oracle
        # gets the lists without it
        keep = [np.isfinite(x[2]) for x in lists]
        cols = [np.ascontiguousarray(x) for k in (la, lb)
                for x in (np.ones(keep[k].sum()), lists[k][1][keep[k]], lists[k][2][keep[k]])]
        L.orc_bf_bin(orc._h, h, cols[0].size, *[oracle_lib._pd(c) for c in cols[:3]],
                     cols[3].size, *[oracle_lib._pd(c) for c in cols[3:]], mx, rot)
    for h in range(len(jobs)):
        np.testing.assert_array_equal(eng.hist(h), orc.hist(h))
