"""Performance cases of the framework: whole calls through its public entry points.

A case is one analysis pass as a user's program runs it: the histograms are
cleared, the pairs of its lists are binned and the histograms are read.  The
kinds (``kind``):

* ``hbt``: HBT pair binning through ``engine.Engine``.  ``path`` says how the
  lists reach the engine: ``device`` (one ``bin_batch`` over device arrays),
  ``host`` (one ``bin_batch`` over host arrays, the drop-in host's way) or
  ``calls`` (a ``bin_same`` / ``bin_mixed`` call per list, host arrays).
  ``n_Kphi`` 0 means no K_phi bins, ``cap`` 0 no pair cap.
* ``serve``: a burst of requests through ``server.Server``.
* ``balance``: balance-function binning through ``bf.BfEngine``.
* ``fit``: Gaussian radii fits through ``radii.Fitter``.

Events come from the package's seeded emission-source model, with the shapes
of its benchmark configurations.
"""
import math

import numpy as np
import torch

from hadronic_afterburner_toolkit_gb300 import bf, engine, radii, server, synth

COLS = ("px", "py", "pz", "E", "x", "y", "z", "t")
PRECISIONS = {"fp64": engine.PRECISION_FP64, "fp32w": engine.PRECISION_FP32W,
              "df64": engine.PRECISION_DF64}
HBARC = 0.197327053       # GeV fm, pair phase
HBARC_FIT = 0.19733       # GeV fm, radii fit
# Share of the candidate pairs that the windows let through (pions of the
# central configuration): what work() takes as pairs that have to be binned.
BINNED = 0.17


def _hbt(name, source, events, mu, oversample, partners, path, **kw):
    c = dict(name=name, kind="hbt", source=source, events=events, mu=mu, oversample=oversample,
             partners=partners, path=path, qnpts=41, q_max=0.15, n_KT=5, n_Kphi=0, boost=True,
             qinv=False, cap=0, precision="fp64")
    c.update(kw)
    return c


def listed():
    return [
        # the smallest analysis: a handful of 80-particle events with K_phi
        # bins and the q_inv histograms on a coarse grid (a quick look, a unit
        # test); launches, copies and synchronisations are all of it
        _hbt("few_events", "pions", 6, 80.0, 6, 2, "host", qnpts=11, n_Kphi=4, qinv=True),
        # event by event: one same-event and one mixed-event call per
        # 1000-particle event, lab-frame q_long (an event loop that bins as it
        # reads)
        _hbt("event_loop", "pions", 24, 1000.0, 1, 3, "calls", boost=False),
        # the small configuration: 100 events of 500 pions, oversampled by 10,
        # 5 partners, one host batch
        _hbt("small_config", "pions", 100, 500.0, 10, 5, "host"),
        # one oversample group of the central configuration (150k particles,
        # 8 x 8 K_T and K_phi bins), the largest plain one
        _hbt("central", "pions", 100, 1500.0, 100, 10, "device", n_KT=9, n_Kphi=8),
        # the same group with FP32 weights (the throughput form)
        _hbt("central_fp32w", "pions", 100, 1500.0, 100, 10, "device", n_KT=9, n_Kphi=8,
             precision="fp32w"),
        # kaon groups of the precision configuration in the double-float form
        _hbt("kaons_df64", "kaons", 300, 250.0, 100, 10, "device", n_KT=9, n_Kphi=8,
             precision="df64"),
        # uneven multiplicities, 20 to 3000 per event, ~50k-particle groups,
        # all in one batch: ragged tiles and many small mixed-event lists
        _hbt("uneven", "uneven", 330, 0.0, 83, 10, "device"),
        # q_inv histograms beside the 3-D ones on a 45k-particle group
        _hbt("qinv", "pions", 30, 1500.0, 30, 10, "device", qinv=True),
        # the reference's default pair cap, which binds on a 60k-particle
        # group without K_phi bins: ordered admission
        _hbt("capped", "pions", 40, 1500.0, 40, 10, "device", cap=30000000),
        # a burst of mixed requests through the serving loop
        dict(name="serving", kind="serve", requests=16, events=120, mu=800.0, partners=1,
             precision="fp64"),
        # pi+ / pi- balance function of 200 events, 8 histograms
        dict(name="balance", kind="balance", events=200, mu=700.0, bnpts=41, rap_max=2.0),
        # radii of 16 events x 4 K_T tables of 41^3 rows, five q cuts each
        dict(name="radii", kind="fit", tables=64, nq=41, q_max=0.15),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["hbt"] * 9 + ["serve", "balance", "fit"])
    if kind == "serve":
        return dict(kind=kind, requests=int(_log(rng, 1, 24)), events=int(_log(rng, 10, 150)),
                    mu=_log(rng, 50, 900), partners=rng.randint(1, 3),
                    precision=rng.choice(["fp64", "fp64", "fp32w"]))
    if kind == "balance":
        return dict(kind=kind, events=int(_log(rng, 1, 300)), mu=_log(rng, 20, 900),
                    bnpts=rng.randint(11, 60), rap_max=rng.uniform(0.8, 3.0))
    if kind == "fit":
        return dict(kind=kind, tables=int(_log(rng, 1, 64)), nq=rng.randint(15, 41),
                    q_max=rng.uniform(0.12, 0.2))
    source = rng.choice(["pions", "pions", "kaons", "uneven"])
    qinv, azimuthal, capped = rng.random() < 0.2, rng.random() < 0.4, rng.random() < 0.15
    mu = _log(rng, 40, 1800) if source != "uneven" else 0.0
    mean = mu or 600.0
    partners = rng.randint(1, 10)
    most = 2.0e9 if qinv or capped else 9.0e9
    want = _log(rng, 2e4, most)
    # particles of one group: half of the wanted pairs or more come from one
    # group, the rest from further ones
    groups = rng.choice([1, 1, 2, 3, 6])
    over = max(1, int(math.sqrt(2.0 * want / groups) / mean))
    while over * partners * mean * mean > want / groups and partners > 1:
        partners -= 1
    n_kphi = rng.randint(3, 8) if azimuthal else 0
    n_kt = rng.randint(3, 9)
    qnpts = rng.choice([11, 16, 21, 31, 41, 41, 51])
    while n_kt * max(1, n_kphi) * qnpts ** 3 > 4_900_000:
        qnpts -= 10
    pairs = groups * 0.5 * (over * mean) ** 2
    path = "device"
    if pairs < 5e8:
        path = rng.choice(["device", "host", "calls" if over * groups <= 40 else "host"])
    return dict(kind="hbt", source=source, events=over * groups, mu=mu, oversample=over,
                partners=partners, path=path, qnpts=qnpts, q_max=rng.uniform(0.1, 0.3),
                n_KT=n_kt, n_Kphi=n_kphi, boost=rng.random() < 0.8, qinv=qinv,
                cap=int(_log(rng, 1e4, 1e7)) if capped and not qinv else 0,
                precision=rng.choice(["fp64", "fp64", "fp32w", "df64"]))


# ------------------------------------------------------------------- inputs

def _events(source, n, mu, seed):
    if source == "uneven":
        return synth.uneven_pions(n_events=n, seed=seed)
    if source == "kaons":
        return synth.central_kaons(n_events=n, mu=mu, seed=seed)
    return synth.central_pions(n_events=n, mu=mu, seed=seed)


def _params(case):
    az = case["n_Kphi"] > 0
    return dict(qnpts=case["qnpts"], q_min=-case["q_max"], q_max=case["q_max"],
                n_KT=case["n_KT"], KT_min=0.0, KT_max=1.0, n_Kphi=case["n_Kphi"] or 8,
                azimuthal_flag=int(az), invariant_radius_flag=int(case["qinv"]),
                long_comoving_boost=int(case["boost"]),
                needed_number_of_pairs=float(case["cap"] or 1e18))


def _jobs(case, seed):
    """Host jobs (the layout of Engine.bin_batch) and the event-plane angle."""
    rng = np.random.default_rng(seed + 1000)
    ev = _events(case["source"], case["events"], case["mu"], seed)
    same, mixed = [], []
    for a in range(0, case["events"], case["oversample"]):
        g = synth.subset(ev, a, min(case["events"], a + case["oversample"]))
        cols = [np.ascontiguousarray(getattr(g, k)) for k in COLS]
        same.append(("same", cols))
        for e in range(g.n_events):
            own = slice(g.offsets[e], g.offsets[e + 1])
            parts = []
            for m in rng.integers(0, g.n_events, size=case["partners"]):
                m = (int(m) + 1) % g.n_events if m == e else int(m)
                phi = rng.uniform(0.0, 2.0 * np.pi)
                c, s = np.cos(phi), np.sin(phi)
                p = slice(g.offsets[m], g.offsets[m + 1])
                px, py = cols[0][p], cols[1][p]
                parts.append((px * c - py * s, px * s + py * c, cols[2][p], cols[3][p]))
            mixed.append(("mixed", [c[own].copy() for c in cols[:4]],
                          [np.concatenate([q[f] for q in parts]) for f in range(4)]))
    return same, mixed, float(rng.uniform(-np.pi, np.pi))


def _requests(case, seed):
    rng = np.random.default_rng(seed)
    grids = np.random.default_rng(case["requests"])  # the grids belong to the case
    reqs = []
    for k in range(case["requests"]):
        n = int(rng.integers(max(2, case["events"] // 3), case["events"] + 1))
        mu = float(rng.uniform(0.3, 1.0)) * case["mu"]
        q_max = float(rng.uniform(0.1, 0.3))
        ev = _events("kaons" if rng.random() < 0.5 else "pions", n, mu, seed * 1000 + k)
        p = dict(qnpts=int(grids.choice([21, 31, 41])), q_min=-q_max, q_max=q_max,
                 n_KT=int(grids.integers(3, 7)), KT_min=0.0, KT_max=1.0,
                 precision=PRECISIONS[case["precision"]])
        reqs.append(([np.ascontiguousarray(getattr(ev, f)) for f in COLS],
                     np.ascontiguousarray(ev.offsets, dtype=np.int64), p, k + 1))
    return reqs


def _balance(case, seed):
    """Species lists (offsets, phi, y) and the job array."""
    rng = np.random.default_rng(seed)
    n, species = case["events"], []
    for k, mon in enumerate((211, -211)):
        g = synth.generate(n, case["mu"], seed=seed * 10 + k, monval=mon, y_max=2.0)
        pt = np.hypot(g.px, g.py)
        keep = (pt >= 0.2) & (pt <= 2.0)
        of = np.repeat(np.arange(n), g.multiplicities())[keep]
        off = np.zeros(n + 1, np.int64)
        np.cumsum(np.bincount(of, minlength=n), out=off[1:])
        species.append((off, np.arctan2(g.py, g.px)[keep],
                        (0.5 * np.log((g.E + g.pz) / (g.E - g.pz)))[keep]))
    lists = [species[0], species[1], species[1], species[0]] * 2
    jobs = []
    for h, (la, lb) in enumerate(((0, 2), (1, 3), (0, 3), (1, 2))):
        for e in range(n):
            jobs.append((h, la, e, lb, e, 0, 0.0))
            jobs.append((4 + h, la, e, 4 + lb, int(rng.integers(n)), 1,
                         float(rng.uniform(0.0, 2.0 * np.pi))))
    return lists, bf.job_array(jobs)


def _tables(case, seed):
    """Eight-column correlation tables: jittered q, a Gaussian source plus noise."""
    rng = np.random.default_rng(seed)
    q = np.linspace(-case["q_max"], case["q_max"], case["nq"])
    ql, qo, qs = [a.ravel() for a in np.meshgrid(q, q, q, indexing="ij")]
    out = []
    for _ in range(case["tables"]):
        lam = rng.uniform(0.3, 0.9)
        r = np.array([rng.uniform(3, 8), rng.uniform(3, 7), rng.uniform(3, 9),
                      rng.uniform(0.6, 2.0), rng.uniform(0.5, 1.6)]) / HBARC_FIT
        t = np.full((qo.size, 8), 1000.0)
        for k, v in enumerate((qo, qs, ql)):
            t[:, k] = v + 0.1 * (q[1] - q[0]) * rng.uniform(-1.0, 1.0, qo.size)
        c0 = lam * np.exp(-(r[0] * t[:, 0]) ** 2 - (r[1] * t[:, 1]) ** 2 - (r[2] * t[:, 2]) ** 2
                          - 2 * t[:, 0] * (t[:, 1] * r[3] ** 2 + t[:, 2] * r[4] ** 2))
        t[:, 7] = 0.004 + 0.03 * c0
        t[:, 6] = c0 + t[:, 7] * rng.standard_normal(qo.size)
        t[:, 4] = 1000.0 * t[:, 6]
        out.append(t)
    return out


def prepare(case, seed):
    if case["kind"] == "serve":
        return case, server.Server(), _requests(case, seed)
    if case["kind"] == "balance":
        return (case, bf.BfEngine(case["bnpts"], case["rap_max"])) + _balance(case, seed)
    if case["kind"] == "fit":
        return case, radii.Fitter(), _tables(case, seed)
    same, mixed, psi = _jobs(case, seed)
    jobs = same + mixed
    if case["path"] == "device":
        jobs = [(j[0],) + tuple([torch.from_numpy(c).cuda() for c in cols] for cols in j[1:])
                for j in jobs]
        torch.cuda.synchronize()
    eng = engine.Engine(precision=PRECISIONS[case["precision"]], **_params(case))
    return case, eng, jobs, psi


# --------------------------------------------------------------------- pass

def run(state):
    case, eng = state[:2]
    if case["kind"] == "serve":
        ids = [eng.submit(cols, off, p, oversample=1, mixed_partners=case["partners"], seed=s)
               for cols, off, p, s in state[2]]
        out = []
        for j in ids:
            eng.wait(j)
            h = eng.result(j)
            eng.release(j)
            out.append(h)
        # one array per quantity: the requests one after another
        return {k: np.concatenate([np.atleast_1d(h[k]) for h in out]) for k in out[0]}
    if case["kind"] == "balance":
        eng.reset()
        eng.bin(state[2], state[3])
        return [eng.hist(k) for k in range(8)]
    if case["kind"] == "fit":
        return eng.fit(state[2])
    eng.reset()
    eng.set_psi_ref(state[3])
    if case["path"] == "calls":
        for j in state[2]:
            if j[0] == "same":
                eng.bin_same(j[1])
            else:
                eng.bin_mixed(j[1], j[2])
    else:
        eng.bin_batch(state[2], device=case["path"] == "device")
    return eng.hist()


# --------------------------------------------------------------------- work

def work(case):
    """Inputs once, outputs once, and per pair that has to be binned the
    operations of its bin and values: FP64 adds, multiplies, divides, roots
    and the cosine of the reference's chain count one each (43 for a
    same-event pair, 31 for a mixed-event one)."""
    if case["kind"] == "balance":
        n = 0.55 * case["mu"]
        pairs = 8 * case["events"] * n * n
        return dict(bytes=2 * 16.0 * case["events"] * n + 8 * 8 * case["bnpts"] * 20.0,
                    flops=6.0 * pairs)
    if case["kind"] == "fit":
        rows = case["tables"] * case["nq"] ** 3
        # the five columns read, the rows of five cuts (0.6 of the table's on
        # average) evaluated in some twelve passes
        return dict(bytes=40.0 * rows, flops=35.0 * 12 * 5 * 0.3 * rows)
    if case["kind"] == "serve":
        n, e = 0.65 * case["mu"], 0.67 * case["events"] * case["requests"]
        pairs = e * n * n * (0.5 + case["partners"])
        bins = case["requests"] * 4 * 31.0 ** 3
        return dict(bytes=64.0 * n * e + 48.0 * bins, flops=37.0 * BINNED * pairs)
    mean = case["mu"] or 600.0
    groups = case["events"] / case["oversample"]
    n = case["oversample"] * mean
    same, mixed = groups * 0.5 * n * n, case["events"] * case["partners"] * mean * mean
    bins = case["n_KT"] * max(1, case["n_Kphi"]) * case["qnpts"] ** 3
    rows = case["events"] * mean * (64.0 + 32.0 + 32.0 * case["partners"])
    return dict(bytes=rows + 48.0 * bins, flops=BINNED * (43.0 * same + 31.0 * mixed))


# -------------------------------------------------------------------- exact

def _pair_block(g, acc, a, b, i0, mixed):
    """Bins the pairs of the rows a (starting at i0) with the rows b, in row
    order, with FP64 tensors in the reference's operand order."""
    ax, bx = [c[:, None] for c in a], [c[None, :] for c in b]
    kx, ky = 0.5 * (ax[0] + bx[0]), 0.5 * (ax[1] + bx[1])
    kp2 = kx * kx + ky * ky
    ok = (kp2 >= g["kt2"][0]) & (kp2 <= g["kt2"][1])
    if not mixed:
        i = torch.arange(i0, i0 + a[0].numel(), device=kp2.device)
        ok &= torch.arange(b[0].numel(), device=kp2.device)[None, :] > i[:, None]
    qt2 = (ax[0] - bx[0]) ** 2 + (ax[1] - bx[1]) ** 2
    far = qt2 > 2.001 * g["hi"] ** 2     # no q_out, q_side inside the window
    keep = ok if g["qinv"] else ok & ~far
    at = torch.nonzero(keep.reshape(-1)).squeeze(1)
    del qt2, ok, keep
    ii, jj = at // b[0].numel(), at % b[0].numel()
    kx, ky, kp2 = kx.reshape(-1)[at], ky.reshape(-1)[at], kp2.reshape(-1)[at]
    far = far.reshape(-1)[at]
    kp = torch.sqrt(kp2)
    ik = ((kp - g["kt_min"]) / g["dkt"]).to(torch.int64)
    A, B = [c[ii] for c in a], [c[jj] for c in b]
    q = [A[f] - B[f] for f in range(4)]
    w = None
    if not mixed:
        d = [A[4 + f] - B[4 + f] for f in range(4)]
        w = torch.cos(g["hbarc_inv"] * (q[3] * d[3] - q[0] * d[0] - q[1] * d[1] - q[2] * d[2]))
        del d
    n = g["qnpts"]
    if g["qinv"]:
        qi = torch.sqrt(-(q[3] * q[3] - q[0] * q[0] - q[1] * q[1] - q[2] * q[2]))
        inside = (qi > g["lo"]) & (qi < g["hi"])
        k = ((torch.where(inside, qi, 0.0) - g["base"]) / g["dq"]).to(torch.int64)
        s = torch.nonzero(inside & (k < n)).squeeze(1)
        flat = (ik * n + k)[s]
        acc["qinv_den" if mixed else "qinv_count"].index_add_(0, flat, torch.ones_like(qi[s]))
        if not mixed:
            acc["qinv_sum"].index_add_(0, flat, qi[s])
            acc["qinv_num"].index_add_(0, flat, w[s])
        del qi, inside, k, s, flat
    cphi, sphi = kx / kp, ky / kp
    qo, qs, ql = q[0] * cphi + q[1] * sphi, q[1] * cphi - q[0] * sphi, q[2]
    if g["boost"]:
        kz, ke = 0.5 * (A[2] + B[2]), 0.5 * (A[3] + B[3])
        ql = ke / torch.sqrt(ke * ke - kz * kz) * (q[2] - kz / ke * q[3])
    ok = ~far
    index = []
    for v in (qo, qs, ql):
        ok &= (v >= g["lo"]) & ((v < g["hi"]) if mixed else (v <= g["hi"]))
        index.append(((torch.where(ok, v, 0.0) - g["base"]) / g["dq"]).to(torch.int64))
        ok &= index[-1] < n
    slot = ik
    if g["n_kphi"]:
        dphi = torch.atan2(ky, kx) - g["psi"]
        for _ in range(2):
            dphi = torch.where(dphi < 0.0, dphi + 2.0 * math.pi, dphi)
            dphi = torch.where(dphi > 2.0 * math.pi, dphi - 2.0 * math.pi, dphi)
        ip = (dphi / g["dkphi"]).to(torch.int64)
        ok &= (ip >= 0) & (ip < g["n_kphi"])
        slot = ik * g["n_kphi"] + ip
    s = torch.nonzero(ok).squeeze(1)
    slot = slot[s]
    if g["cap"]:
        # admission in pair order: a slot takes pairs until its count passes
        # the cap
        count = acc["den_count" if mixed else "num_count"]
        for m in range(count.numel()):
            t = torch.nonzero(slot == m).squeeze(1)
            room = max(0, g["cap"] + 1 - int(count[m]))
            count[m] += min(room, t.numel())
            slot[t[room:]] = -1
        s, slot = s[slot >= 0], slot[slot >= 0]
    flat = ((slot * n + index[0][s]) * n + index[1][s]) * n + index[2][s]
    acc["den" if mixed else "count"].index_add_(0, flat, torch.ones_like(kp2[s]))
    if not mixed:
        for k, v in (("q_out", qo), ("q_side", qs), ("q_long", ql), ("num", w)):
            acc[k].index_add_(0, flat, v[s])


def _exact_hbt(case, seed):
    p = _params(case)
    same, mixed, psi = _jobs(case, seed)
    dq = (p["q_max"] - p["q_min"]) / (p["qnpts"] - 1)
    n_slots = p["n_KT"] * max(1, case["n_Kphi"])
    g = dict(qnpts=p["qnpts"], dq=dq, lo=p["q_min"] - dq / 2. + 1e-8, hi=p["q_max"] + dq / 2. - 1e-8,
             base=p["q_min"] - dq / 2., kt_min=p["KT_min"],
             dkt=(p["KT_max"] - p["KT_min"]) / (p["n_KT"] - 1),
             kt2=(p["KT_min"] * p["KT_min"], p["KT_max"] * p["KT_max"]), n_kphi=case["n_Kphi"],
             dkphi=2 * math.pi / p["n_Kphi"], psi=psi, hbarc_inv=1. / HBARC,
             qinv=case["qinv"], boost=case["boost"], cap=case["cap"])
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    bins, nq = n_slots * p["qnpts"] ** 3, p["n_KT"] * p["qnpts"]
    new = lambda size: torch.zeros(size, dtype=torch.float64, device=dev)  # noqa: E731
    acc = {k: new(bins) for k in ("count", "q_out", "q_side", "q_long", "num", "den")}
    acc.update({k: new(nq) for k in ("qinv_sum", "qinv_num", "qinv_count", "qinv_den")})
    acc.update({k: torch.zeros(n_slots, dtype=torch.int64, device=dev)
                for k in ("num_count", "den_count")})
    total = [0, 0]
    for j in same + mixed:
        is_mixed = j[0] == "mixed"
        a = [torch.from_numpy(np.ascontiguousarray(c)).to(dev) for c in j[1]]
        b = [torch.from_numpy(np.ascontiguousarray(c)).to(dev) for c in j[2]] if is_mixed else a
        na, nb = a[0].numel(), b[0].numel()
        total[is_mixed] += na * nb if is_mixed else na * (na - 1) // 2
        step = max(1, (1 << 26) // max(1, nb))
        for i0 in range(0, na, step):
            # columns before the first row hold no pair of a same-event list
            lo = 0 if is_mixed else i0
            _pair_block(g, acc, [c[i0:i0 + step] for c in a], [c[lo:] for c in b], i0 - lo,
                        is_mixed)
    out = {k: acc[k].cpu().numpy() for k in ("count", "q_out", "q_side", "q_long", "num", "den",
                                             "qinv_sum", "qinv_num", "qinv_count", "qinv_den")}
    for key, h, n in (("ctr_num", "count", n_slots), ("ctr_den", "den", n_slots),
                      ("ctr_num_qinv", "qinv_count", p["n_KT"]),
                      ("ctr_den_qinv", "qinv_den", p["n_KT"])):
        out[key] = out[h].reshape(n, -1).sum(axis=1).astype(np.int64)
    out.update(anomalies=0, pairs_same=total[0], pairs_mixed=total[1])
    return out


def _exact_balance(case, seed):
    lists, jobs = _balance(case, seed)
    drap = 2. * abs(case["rap_max"]) / (case["bnpts"] - 1)
    ymin, dphi, pmin = -abs(case["rap_max"]) - 0.5 * drap, 2. * math.pi / 20, -math.pi / 2.
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    cols = [[torch.from_numpy(c).to(dev) for c in lst[1:]] for lst in lists]
    acc = torch.zeros((8, case["bnpts"] * 20), dtype=torch.int64, device=dev)
    for hist, la, ea, lb, eb, mixed, rot in jobs.tolist():
        a = slice(lists[la][0][ea], lists[la][0][ea + 1])
        b = slice(lists[lb][0][eb], lists[lb][0][eb + 1])
        d = cols[la][0][a][:, None] - cols[lb][0][b][None, :]
        if mixed:
            d = d + rot
        ip = torch.remainder(torch.floor((d - pmin) / dphi).to(torch.int64), 20)
        dy = cols[la][1][a][:, None] - cols[lb][1][b][None, :]
        iy = ((dy - ymin) / drap).to(torch.int64)
        ok = (dy.abs() >= 1e-10) & (dy >= ymin) & (iy < case["bnpts"])
        acc[hist] += torch.bincount((iy * 20 + ip)[ok], minlength=case["bnpts"] * 20)
    return [h.reshape(case["bnpts"], 20).cpu().numpy().astype(np.float64) for h in acc]


def _exact_fit(case, seed):
    """The least-squares minimum of every (table, cut): damped steps, then
    Gauss-Newton until it stands still."""
    cuts = (0.05, 0.075, 0.1, 0.125, 0.15)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    out = np.empty((case["tables"], len(cuts), 13))
    for k, t in enumerate(_tables(case, seed)):
        t = torch.from_numpy(t).to(dev)
        qabs = torch.sqrt(t[:, 0] ** 2 + t[:, 1] ** 2 + t[:, 2] ** 2)
        for m, cut in enumerate(cuts):
            r = t[(qabs > 0.0) & (qabs < cut)]
            q = torch.stack([r[:, 0] ** 2, r[:, 1] ** 2, r[:, 2] ** 2, 2 * r[:, 0] * r[:, 1],
                             2 * r[:, 0] * r[:, 2]])
            weight = 1.0 / (r[:, 7] + 1e-15)

            def at(p):
                e = torch.exp(-((p[1:] / HBARC_FIT) ** 2 @ q))
                jac = torch.cat([e[None], -2 * p[0] * e * p[1:, None] / HBARC_FIT ** 2 * q])
                res, jac = weight * (p[0] * e - r[:, 6]), weight * jac
                return (res @ res), jac @ res, jac @ jac.T

            p = torch.tensor([1.0, 5.0, 5.0, 5.0, 0.1, 0.1], dtype=torch.float64, device=dev)
            chi2, grad, hess = at(p)
            mu = 1e-3
            for it in range(60):
                step = torch.linalg.solve(hess + mu * torch.diag(torch.diag(hess)), -grad)
                new = at(p + step)
                if bool(new[0] <= chi2):
                    p, (chi2, grad, hess), mu = p + step, new, mu * 0.1
                    if it > 8 and float((step / p).abs().max()) < 1e-9:
                        break
                else:
                    mu *= 10.0
            for _ in range(12):
                p = p + torch.linalg.solve(hess, -grad)
                chi2, grad, hess = at(p)
            err = torch.sqrt(torch.diag(torch.linalg.inv(hess)))
            out[k, m, 0] = cut
            out[k, m, 1::2], out[k, m, 2::2] = p.cpu().numpy(), err.cpu().numpy()
    return out


def exact(case, seed):
    if case["kind"] == "hbt":
        # the FP64 chain over every pair
        return _exact_hbt(case, seed)
    if case["kind"] == "balance":
        return _exact_balance(case, seed)
    if case["kind"] == "fit":
        return _exact_fit(case, seed)
    return None  # the server draws its own partners and angles
