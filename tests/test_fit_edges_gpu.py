"""The batched fits at the edges of their row selection (4096 rows to a block)
and of their work items (8192 kept rows, units of 32 lanes), against the scipy
oracle; the kept rows are counted exactly, rows with |q| equal to a cut among
them.  Tolerances: tests/test_fit_gpu.py."""
import os
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(os.path.dirname(HERE), "oracle"))

from test_fit_gpu import _close  # noqa: E402

pytestmark = pytest.mark.gpu


def _table(n, nq, rng):
    """n random rows of a grid whose nodes lie on the cuts."""
    q = np.linspace(-0.15, 0.15, nq)
    ql, qo, qs = [a.ravel() for a in np.meshgrid(q, q, q, indexing="ij")]
    t = np.zeros((qo.size, 8))
    t[:, 0], t[:, 1], t[:, 2] = qo, qs, ql
    r = np.array([5.0, 4.5, 5.5, 1.4, 1.2]) / 0.19733
    c = 0.6 * np.exp(-(r[0] * qo) ** 2 - (r[1] * qs) ** 2 - (r[2] * ql) ** 2
                     - 2 * qo * (qs * r[3] ** 2 + ql * r[4] ** 2))
    t[:, 7] = 0.002 + 0.01 * c
    t[:, 6] = c + t[:, 7] * rng.standard_normal(qo.size)
    return t[np.sort(rng.permutation(qo.size)[:n])]


@pytest.mark.parametrize("n", [400, 4095, 4096, 4097, 8193, 15700])
def test_row_counts_and_fits_at_edges(n):
    import fit_radii
    from hadronic_afterburner_toolkit_gb300 import radii
    rng = np.random.default_rng(n)
    tabs = [_table(n, 25, rng), np.zeros((0, 8)), _table(n // 2, 25, rng)]
    cuts = [0.1, 0.125, 0.15, 0.3]
    f = radii.Fitter()
    got = f.fit(tabs, q_cut_max_list=cuts)
    for k in (0, 2):
        t = tabs[k]
        qabs = np.sqrt(t[:, 0] ** 2. + t[:, 1] ** 2. + t[:, 2] ** 2.)
        want = [int(((qabs > 0.0) & (qabs < c)).sum()) for c in cuts]
        assert f.last["n_points"][k].tolist() == want
        # the radii enter squared: either sign is the same minimum
        _close(np.abs(got[k]), np.abs(fit_radii.fit_table(t, q_cut_max_list=cuts)))
    assert (f.last["n_points"][1] == 0).all() and (f.last["status"][1] == 3).all()
