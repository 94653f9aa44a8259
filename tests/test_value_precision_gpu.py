"""q_out, q_side and q_long of binned pairs to the precision of double-float
arithmetic on exact FP64 differences, 2^-43 of the window a pair, against
extended precision: on ordinary grids and on grids whose bins are far smaller
than the momenta (where a fixed-point momentum's 2^-57 GeV would show), for
momenta of a few MeV and of several GeV."""
import numpy as np
import pytest

from hadronic_afterburner_toolkit_gb300 import engine

pytestmark = pytest.mark.gpu
LD = np.longdouble
N = 240


def particles(p_center, spread, seed):
    rng = np.random.default_rng(seed)
    px, py, pz = (c + spread * rng.uniform(-1.0, 1.0, N) for c in p_center)
    E = np.sqrt(0.13957 ** 2 + px * px + py * py + pz * pz)
    return [np.ascontiguousarray(c) for c in (px, py, pz, E, *rng.normal(0.0, 5.0, (4, N)))]


def exact(cols, boost, p):
    """Per-bin counts and sums (one K_T slot), pairs i < j."""
    i, j = np.triu_indices(N, 1)
    x, y, z, E = (c.astype(LD) for c in cols[:4])
    dx, dy, dz, dE = (c[i] - c[j] for c in (x, y, z, E))
    sx, sy = x[i] + x[j], y[i] + y[j]
    k = np.sqrt(sx * sx + sy * sy)
    m, q = E - z, E + z
    q_long = (m[j] * q[i] - m[i] * q[j]) / np.sqrt((m[i] + m[j]) * (q[i] + q[j])) if boost else dz
    v = [(dx * sx + dy * sy) / k, (dy * sx - dx * sy) / k, q_long]
    n, dq = p["qnpts"], LD(p["q_max"] - p["q_min"]) / (p["qnpts"] - 1)
    t = [(a - LD(p["q_min"])) / dq + LD(0.5) for a in v]
    # the window ends 1e-8 GeV inside the outer bins' edges
    inset = LD(1e-8) / dq
    ok = np.logical_and.reduce([(a > inset) & (a < n - inset) for a in t])
    # no pair so close to an edge that FP64 could bin it elsewhere
    assert min(np.abs(a[ok] - np.rint(a[ok])).min() for a in t) > 1e-9
    b = [a[ok].astype(int) for a in t]
    flat = (b[0] * n + b[1]) * n + b[2]
    sums = []
    for a in v:
        s = np.zeros(n ** 3, LD)
        np.add.at(s, flat, a[ok])
        sums.append(s)
    return np.bincount(flat, minlength=n ** 3), sums


@pytest.mark.parametrize("precision", [engine.PRECISION_FP64, engine.PRECISION_DF64])
@pytest.mark.parametrize("boost", [0, 1])
@pytest.mark.parametrize("p_center,q_max", [((0.03, -0.02, 0.01), 0.15), ((0.03, -0.02, 0.01), 2e-5),
                                            ((0.3, 0.2, 0.3), 1e-4), ((7.0, 5.0, 3.0), 0.15),
                                            ((7.0, 5.0, 3.0), 2e-3)])
def test_sums_to_double_float(p_center, q_max, boost, precision):
    p = dict(qnpts=7, q_min=-q_max, q_max=q_max, n_KT=2, KT_min=0.0, KT_max=40.0, n_Kphi=4,
             azimuthal_flag=0, invariant_radius_flag=0, long_comoving_boost=boost,
             needed_number_of_pairs=1e18)
    cols = particles(p_center, min(q_max, 0.02) if p_center[0] < 0.1 else q_max, 17)
    count, sums = exact(cols, boost, p)
    eng = engine.Engine(precision=precision, **p)
    eng.bin_same(cols)
    h = eng.hist()
    eng.close()
    assert np.array_equal(h["count"][:343], count) and count.sum() > 1000
    for s, k in zip(sums, ("q_out", "q_side", "q_long")):
        # a pair's value, and n additions of the sum
        tol = count * q_max * (2.0 ** -43 + count * 2.0 ** -53)
        assert np.all(np.abs(h[k][:343] - s) <= tol), k


def test_fine_and_wide_grids_served_together():
    """Analyses of both kinds of grid in the serving loop's shared launches."""
    from hadronic_afterburner_toolkit_gb300 import server
    cols = particles((0.03, -0.02, 0.01), 2e-5, 17)
    grids = [dict(qnpts=7, q_min=-q, q_max=q, n_KT=2, KT_min=0.0, KT_max=40.0)
             for q in (0.15, 2e-5, 0.05, 1e-5)]
    with server.Server(max_in_flight=2) as srv:
        jobs = [srv.submit(cols, np.array([0, N]), g, mixed_partners=1, seed=3) for g in grids * 4]
        for j in jobs:
            srv.wait(j)
        for j, g in zip(jobs, grids * 4):
            count, sums = exact(cols, 1, g)
            h = srv.result(j)
            assert np.array_equal(h["count"][:343], count) and count.sum() > 1000
            for s, k in zip(sums, ("q_out", "q_side", "q_long")):
                tol = count * g["q_max"] * (2.0 ** -43 + count * 2.0 ** -53)
                assert np.all(np.abs(h[k][:343] - s) <= tol), k
