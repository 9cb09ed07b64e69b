"""Performance cases: the calls a user of this library makes, over the sizes,
types and modes they come in.

Kinds (each one public call of ``opendba_b200.api``, or the pair of calls a
device-side program makes):

* ``medoid``  -- ``medoid_pass_host``: host series in, z-normalisation, all
  pair distances, medoid, distances and normalisation figures back.
* ``pairs``   -- ``pairwise`` and ``medoid`` on series that already live on the
  device (a sweep of parameters, a shard's range, a second pass).
* ``round``   -- ``dba_round``: one averaging round of all members against the
  current centroid; repeated up to 250 times per average.
* ``stripe``  -- ``dba_round`` in stripe mode: members too long to keep a path.
* ``segment`` -- ``segment_host``: raw signal to segment medians.
* ``jobs``    -- ``dba_jobs``: many whole averages (normalise, medoid, rounds).
* ``serve``   -- one read-against-centroids query through ``Server``.

Signals are nanopore-like step signals or Gaussian random walks from
``opendba_b200.synth``; the members of an average are noisy, time-warped copies
of one signal, as reads of one molecule are.
"""
import math

import numpy as np
import torch

from opendba_b200 import api, synth

_F = {"f32": np.float32, "f64": np.float64}


def listed():
    return [
        # Medoid pass over reads (the headline configuration's lengths) from
        # host memory: the call that dominates averaging a set of reads.
        {"name": "medoid_reads", "kind": "medoid", "n": 300, "lo": 2000, "hi": 8000,
         "dtype": "f32", "os": 0, "oe": 0, "data": "reads"},
        # The plain averaging configuration: a few dozen short series, open end.
        {"name": "medoid_walks", "kind": "medoid", "n": 64, "lo": 512, "hi": 1024,
         "dtype": "f32", "os": 0, "oe": 1, "data": "walks"},
        # The smallest call: a handful of short series already on the device.
        {"name": "pairs_tiny", "kind": "pairs", "n": 8, "lo": 150, "hi": 400,
         "dtype": "f32", "os": 0, "oe": 0, "data": "walks"},
        # Double precision, the other build of the command line.
        {"name": "pairs_double", "kind": "pairs", "n": 100, "lo": 1000, "hi": 4000,
         "dtype": "f64", "os": 0, "oe": 0, "data": "reads"},
        # Few long raw signals (whole reads without segmentation).
        {"name": "pairs_long", "kind": "pairs", "n": 8, "lo": 40000, "hi": 80000,
         "dtype": "f32", "os": 0, "oe": 0, "data": "reads"},
        # One averaging round of a few hundred reads.
        {"name": "round_reads", "kind": "round", "n": 400, "lo": 3000, "hi": 8000,
         "dtype": "f32", "os": 0, "oe": 0, "data": "reads"},
        # One round of the plain averaging configuration, open end.
        {"name": "round_walks", "kind": "round", "n": 64, "lo": 512, "hi": 1024,
         "dtype": "f32", "os": 0, "oe": 1, "data": "walks"},
        # One round in double.
        {"name": "round_double", "kind": "round", "n": 100, "lo": 1000, "hi": 4000,
         "dtype": "f64", "os": 0, "oe": 0, "data": "reads"},
        # Stripe mode: very long members, no path held in memory.
        {"name": "round_stripe", "kind": "stripe", "n": 3, "lo": 40000, "hi": 80000,
         "dtype": "f32", "os": 0, "oe": 0, "data": "reads", "rows": 1024},
        # Segmentation of raw signal before averaging.
        {"name": "segment_raw", "kind": "segment", "n": 8, "lo": 100000, "hi": 400000,
         "dtype": "f32", "minseg": 4, "data": "reads"},
        # Whole averages: many independent clusters of reads at once, open end.
        {"name": "jobs_clusters", "kind": "jobs", "jobs": 24, "n_lo": 8, "n_hi": 48,
         "lo": 200, "hi": 2000, "dtype": "f32", "os": 0, "oe": 1, "rounds": 12, "data": "reads"},
        # A serving query: a batch of reads against resident centroids.
        {"name": "serve_query", "kind": "serve", "n": 16, "lo": 500, "hi": 50000,
         "centroids": 32, "clen": 4000, "dtype": "f32", "os": 0, "oe": 0, "data": "reads"},
    ]


# ---- drawn cases ---------------------------------------------------------------

_CELL_CAP = 1.1e12       # float: the listed medoid pass
_CELL_CAP_F64 = 2.5e11   # double runs at about a quarter of float's rate


def _logu(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mode(rng):
    """Global most of the time, then open end, then the other two."""
    u = rng.random()
    return (0, 0) if u < 0.5 else (0, 1) if u < 0.8 else (1, 0) if u < 0.9 else (1, 1)


def _lens(rng, lo_min, hi_max):
    hi = _logu(rng, 2 * lo_min, hi_max)
    lo = max(lo_min, int(hi * rng.uniform(0.25, 0.9)))
    return lo, hi


def draw(rng):
    kind = rng.choice(["medoid", "medoid", "pairs", "pairs", "round", "round", "round", "stripe",
                       "segment", "jobs", "serve"])
    dtype = "f64" if rng.random() < 0.25 else "f32"
    os_, oe = _mode(rng)
    data = rng.choice(["reads", "walks"])
    case = {"kind": kind, "dtype": dtype, "os": os_, "oe": oe, "data": data}
    cap = _CELL_CAP if dtype == "f32" else _CELL_CAP_F64
    if kind == "medoid" or (kind == "pairs" and rng.random() < 0.7):
        lo, hi = _lens(rng, 150, 8000)
        n = _logu(rng, 4, 300)
        while n > 4 and 0.5 * n * n * (0.5 * (lo + hi)) ** 2 > cap:
            n -= 1
        case.update(n=n, lo=lo, hi=hi)
    elif kind == "pairs":
        lo, hi = _lens(rng, 20000, 100000)
        n = rng.randint(3, 10)
        while n > 3 and 0.5 * n * n * (0.5 * (lo + hi)) ** 2 > cap:
            n -= 1
        case.update(n=n, lo=lo, hi=hi)
    elif kind == "round":
        lo, hi = _lens(rng, 200, 8000)
        n = _logu(rng, 4, 400)
        while n > 4 and n * (0.5 * (lo + hi)) ** 2 > 1.4e10:
            n -= 1
        case.update(n=n, lo=lo, hi=hi)
    elif kind == "stripe":
        lo, hi = _lens(rng, 10000, 80000)
        n = rng.randint(1, 4)
        while n > 1 and n * (0.5 * (lo + hi)) ** 2 > 1.1e10:
            n -= 1
        case.update(n=n, lo=lo, hi=hi, rows=rng.choice([1024, 2048, 4096]))
    elif kind == "segment":
        lo, hi = _lens(rng, 5000, 400000)
        case.update(n=rng.randint(1, 8), lo=lo, hi=hi, minseg=rng.choice([3, 4, 5, 6, 8]))
        del case["os"], case["oe"]
    elif kind == "jobs":
        lo, hi = _lens(rng, 100, 2000)
        n_hi = rng.randint(4, 48)
        case.update(jobs=_logu(rng, 1, 24), n_lo=max(2, n_hi // 6), n_hi=n_hi, lo=lo, hi=hi,
                    rounds=rng.randint(2, 12))
    else:
        lo, hi = _lens(rng, 500, 50000)
        case.update(n=_logu(rng, 1, 16), lo=lo, hi=hi, centroids=rng.randint(1, 32),
                    clen=_logu(rng, 500, 4000), dtype="f32")
    return case


# ---- inputs ----------------------------------------------------------------------

def _rng(seed):
    return np.random.default_rng([0x0DBA, int(seed)])


def _shape_rng(case):
    """Lengths depend on the case alone, so that every seed is the same work."""
    key = [0x0DBA] + [int(case[k]) for k in sorted(case) if isinstance(case[k], (int, bool))]
    return np.random.default_rng(key)


def _lengths(case):
    r = _shape_rng(case)
    if case["kind"] == "jobs":
        counts = r.integers(case["n_lo"], case["n_hi"] + 1, size=case["jobs"])
        return [np.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"] + 1), size=int(c)))
                .astype(np.int64) for c in counts]
    if case["kind"] == "serve":
        return np.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"] + 1),
                                size=case["n"])).astype(np.int64)
    lens = r.integers(case["lo"], case["hi"] + 1, size=case["n"])
    return np.sort(lens)  # an averaging run sorts its series by length first


def _signals(rng, lens, data, dtype):
    """Unrelated raw signals."""
    if data == "reads":
        return synth.step_signals(rng, lens, 90.0, 12.0, 10.0, 2.0, dtype=dtype)
    return [np.cumsum(rng.standard_normal(int(L))).astype(dtype) for L in lens]


def _copies(rng, lens, data, dtype):
    """Noisy time-warped copies of one signal."""
    k = max(4, int(np.mean(lens)) // 10)
    if data == "reads":
        levels = rng.normal(90.0, 12.0, size=k)
    else:
        levels = np.cumsum(rng.standard_normal(k) * 3.0)
    noise = 2.0 if data == "reads" else 0.5
    out = []
    for L in lens:
        L = int(L)
        edges = np.cumsum(rng.geometric(0.1, size=k).astype(np.float64))
        idx = np.searchsorted(edges * (L / edges[-1]), np.arange(L) + 0.5)
        out.append((levels[np.minimum(idx, k - 1)] + rng.normal(0.0, noise, size=L)).astype(dtype))
    return out


def _host_inputs(case, seed):
    """The host series of a case (raw), or (members, centroid index) parts."""
    rng = _rng(seed)
    lens = _lengths(case)
    dt = _F[case["dtype"]]
    kind = case["kind"]
    if kind == "jobs":
        return [_copies(rng, job, case["data"], dt) for job in lens]
    if kind in ("round", "stripe"):
        return synth.znorm_host(_copies(rng, lens, case["data"], dt))
    if kind == "pairs":
        return synth.znorm_host(_signals(rng, lens, case["data"], dt))
    if kind == "serve":
        reads = synth.znorm_host(_signals(rng, lens, case["data"], dt))
        cents = synth.znorm_host(_signals(rng, [case["clen"]] * case["centroids"], case["data"], dt))
        return reads, cents
    return _signals(rng, lens, case["data"], dt)


def prepare(case, seed):
    kind = case["kind"]
    host = _host_inputs(case, seed)
    if kind == "medoid":
        flat, _, lens = api.pack_host(host)
        pinned = torch.from_numpy(flat).pin_memory()
        return {"case": case, "flat": pinned.numpy(), "pinned": pinned, "lens": lens}
    if kind == "pairs":
        return {"case": case, "ds": api.DeviceSeries.from_host(host)}
    if kind in ("round", "stripe"):
        ds = api.DeviceSeries.from_host(host)
        cen = torch.from_numpy(np.ascontiguousarray(host[len(host) // 2])).cuda()
        return {"case": case, "ds": ds, "centroid": cen}
    if kind in ("segment", "jobs"):
        return {"case": case, "host": host}
    reads, cents = host
    srv = api.Server(_F[case["dtype"]], hbm_budget_bytes=2 << 30)
    ids = [srv.add_centroid(c) for c in cents]
    return {"case": case, "server": srv, "ids": ids, "reads": reads}


def _padded(rows, width):
    """Ragged results as a zero-padded matrix and their lengths."""
    out = np.zeros((len(rows), width), dtype=rows[0].dtype)
    for k, row in enumerate(rows):
        out[k, :len(row)] = row
    return out, np.array([len(row) for row in rows])


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "medoid":
        return api.medoid_pass_host(None, case["os"], case["oe"], norm=1, flat=state["flat"],
                                    lens=state["lens"])
    if kind == "pairs":
        d = api.pairwise(state["ds"], case["os"], case["oe"])
        sos, med = api.medoid(d, state["ds"])
        return d, sos, med
    if kind in ("round", "stripe"):
        mean, counts, delta, _ = api.dba_round(state["centroid"], state["ds"], case["os"], case["oe"],
                                               stripe_rows=case.get("rows"))
        return mean, counts, delta
    if kind == "segment":
        return _padded(api.segment_host(state["host"], case["minseg"]), max(len(s) for s in state["host"]) // 2)
    if kind == "jobs":
        res = api.dba_jobs(state["host"], [case["os"] | (case["oe"] << 1)] * case["jobs"], norm=1,
                           max_rounds=case["rounds"])
        longest = max(len(s) for job in state["host"] for s in job)
        return _padded([r["centroid"] for r in res], longest) + (
            np.array([r["medoid"] for r in res]), np.array([r["rounds"] for r in res]),
            np.array([r["delta"] for r in res]))
    srv = state["server"]
    rid = srv.submit_query(state["reads"], state["ids"], case["os"], case["oe"])
    if srv.wait(rid) != 1:
        raise RuntimeError("the query failed")
    return srv.take(rid)["result"]


# ---- work ------------------------------------------------------------------------

def _pair_cells(lens):
    lens = np.asarray(lens, dtype=np.float64)
    return float((lens.sum() ** 2 - (lens * lens).sum()) / 2.0)


def work(case):
    """A DTW cell is a difference, a multiply-add and two minima: 5 operations.
    Bytes: every input sample once, every result once."""
    item = 4 if case["dtype"] == "f32" else 8
    kind = case["kind"]
    lens = _lengths(case)
    if kind in ("medoid", "pairs"):
        n = case["n"]
        return {"bytes": float(lens.sum()) * item + 0.5 * n * (n - 1) * item + 8.0 * n,
                "flops": 5.0 * _pair_cells(lens)}
    if kind in ("round", "stripe"):
        lc = float(lens[len(lens) // 2])
        return {"bytes": float(lens.sum()) * item + lc * (2 * item + 4),
                "flops": 5.0 * float(lens.sum()) * lc}
    if kind == "segment":
        # the input, one median per three or so samples, and per 256-point block
        # the costs of all point pairs (a difference, a square and a division)
        points = float(lens.sum()) / ((case["minseg"] + 2) // 3)
        return {"bytes": float(lens.sum()) * item * (1 + 1.0 / case["minseg"]),
                "flops": points * 128 * 3.0}
    if kind == "jobs":
        tot = sum(float(j.sum()) for j in lens)
        cells = sum(_pair_cells(j) + float(j.sum()) * float(np.median(j)) for j in lens)
        return {"bytes": tot * item, "flops": 5.0 * cells}
    cells = float(lens.sum()) * case["centroids"] * case["clen"]
    return {"bytes": (float(lens.sum()) + case["centroids"] * case["clen"] +
                      case["n"] * case["centroids"]) * item, "flops": 5.0 * cells}


# ---- 64-bit values ----------------------------------------------------------------

class _Dtw:
    """The DTW matrices of many pairs at once in float64, one anti-diagonal per
    step: rows from ``xs[p]``, columns from ``ys[p]``; a cell costs the squared
    difference plus the least of up, left and diagonal; with ``oe`` the last
    row's moves to the right are free."""

    def __init__(self, xs, ys, oe, moves):
        dev = "cuda"
        self.m = np.array([len(x) for x in xs])
        self.n = np.array([len(y) for y in ys])
        p, big_m, big_n = len(xs), int(self.m.max()), int(self.n.max())
        inf = float("inf")
        xp = torch.full((p, big_m + 2 * big_n), inf, dtype=torch.float64, device=dev)
        y = torch.zeros((p, big_n), dtype=torch.float64, device=dev)
        for i in range(p):
            xp[i, big_n:big_n + self.m[i]] = xs[i]
            y[i, :self.n[i]] = ys[i]
        xr = xp.flip(1).contiguous()
        ends = {}
        for i in range(p):
            ends.setdefault(int(self.m[i] + self.n[i] - 2), []).append(i)
        cost = torch.empty(p, dtype=torch.float64, device=dev)
        diags = big_m + big_n - 1
        self.codes = torch.zeros((diags, p, big_n), dtype=torch.int8, device=dev) if moves else None
        if oe:
            jj = torch.arange(big_n, device=dev)[None, :]
            mm = torch.from_numpy(self.m).to(dev)[:, None]
        # column -1 of each diagonal is absent: one leading infinity
        a = torch.full((p, big_n + 1), inf, dtype=torch.float64, device=dev)
        b, c = a.clone(), a.clone()
        b[:, 0] = 0.0  # the virtual corner, diagonal of cell (0, 0)
        prev1, prev2, cur = a, b, c
        for k in range(diags):
            s = big_m + big_n - 1 - k
            d = xr[:, s:s + big_n] - y
            d.mul_(d)
            up, left, diag = prev1[:, 1:], prev1[:, :-1], prev2[:, :-1]
            out = cur[:, 1:]
            best = torch.minimum(up, diag)
            if oe:
                top = jj == (k + 1 - mm)
                side = torch.where(top & (mm > 1), left - d, left)
                torch.minimum(best, side, out=best)
            else:
                side = left
                torch.minimum(best, left, out=best)
            if moves:
                # diagonal over up over right
                code = torch.where(diag == best, 1, torch.where(up == best, 3, 2))
                self.codes[k] = code
            torch.add(d, best, out=out)
            if k in ends:
                i = torch.tensor(ends[k], device=dev)
                j = torch.from_numpy(self.n[ends[k]]).to(dev)
                cost[i] = cur[i, j]
            if k == 0:
                b[:, 0] = inf
            prev1, prev2, cur = cur, prev1, prev2
            cur[:, 0] = inf
        self.cost = cost


def _seconds(xs_lens, ys_lens, moves):
    diags = float(np.max(xs_lens) + np.max(ys_lens))
    vec = float(len(xs_lens)) * float(np.max(ys_lens))
    return diags * max(1.2e-4 if moves else 0.8e-4, vec * 8 * (16 if moves else 10) / 4.5e12)


def _exact_dists(xs, ys, os_, oe):
    """Pair distances, or None where the plain matrix is not the definition: the
    library follows its reference in every 1024-column block of an open
    alignment, and an open start has rules of its own."""
    if os_ or (oe and max(len(y) for y in ys) > 1024):
        return None
    if _seconds([len(x) for x in xs], [len(y) for y in ys], False) > 18:
        return None
    w = _Dtw(xs, ys, oe, False)
    d = torch.sqrt(w.cost)
    if oe:
        d = d / torch.from_numpy(w.m.astype(np.float64)).to(d.device)
    return d


def _tensors(series):
    return [torch.from_numpy(np.asarray(s, dtype=np.float64)).cuda() for s in series]


def _exact_pairs(series, os_, oe):
    n = len(series)
    s, j = np.triu_indices(n, 1)
    return _exact_dists([series[i] for i in s], [series[i] for i in j], os_, oe)


def _exact_round(case, seed):
    if case["os"] or (case["oe"] and case["hi"] > 1024):
        return None
    host = _host_inputs(case, seed)
    series = _tensors(host)
    cen = series[len(series) // 2]
    lc, oe = len(cen), case["oe"]
    flip = [bool(oe and lc < len(s)) for s in series]
    xs = [cen if f else s for s, f in zip(series, flip)]
    ys = [s if f else cen for s, f in zip(series, flip)]
    ml, nl = [len(x) for x in xs], [len(y) for y in ys]
    if (_seconds(ml, nl, True) + 2e-4 * (max(ml) + max(nl)) > 18 or
            float(max(ml) + max(nl)) * len(ml) * max(nl) > 5e10):
        return None
    w = _Dtw(xs, ys, oe, True)
    dev = cen.device
    p = len(xs)
    idx = torch.arange(p, device=dev)
    r = torch.from_numpy(w.m - 1).to(dev)
    c = torch.from_numpy(w.n - 1).to(dev)
    top = r.clone()
    flip_t = torch.tensor(flip, device=dev)
    data = torch.zeros((p, max(len(s) for s in series)), dtype=torch.float64, device=dev)
    for i, s in enumerate(series):
        data[i, :len(s)] = s
    total = torch.zeros(lc, dtype=torch.float64, device=dev)
    count = torch.zeros(lc, dtype=torch.float64, device=dev)
    alive = torch.ones(p, dtype=torch.bool, device=dev)
    for _ in range(max(ml) + max(nl)):
        code = w.codes[r + c, idx, c].to(torch.int64)
        at_start = (r == 0) & (c == 0)
        code = torch.where(r == 0, 2, code)
        free = (code == 2) & (r == top) & (top > 0) if oe else torch.zeros_like(alive)
        take = (alive & (~free | at_start)).to(torch.float64)
        ci, mi = torch.where(flip_t, r, c), torch.where(flip_t, c, r)
        total.index_add_(0, ci, data[idx, mi] * take)
        count.index_add_(0, ci, take)
        alive = alive & ~at_start
        r = torch.where(alive & (code != 2), r - 1, r)
        c = torch.where(alive & (code != 3), c - 1, c)
    mean = total / count
    del w
    torch.cuda.empty_cache()
    return mean, None, float((mean - cen).abs().max())


def exact(case, seed):
    kind = case["kind"]
    if kind in ("medoid", "pairs"):
        host = _host_inputs(case, seed)
        if kind == "medoid":
            raw = [np.asarray(s, dtype=np.float64) for s in host]
            means = np.array([x.mean() for x in raw])
            sigmas = np.array([x.std() for x in raw])
            host = [(x - m) / (s if s != 0 else 1.0) for x, m, s in zip(raw, means, sigmas)]
        d = _exact_pairs(_tensors(host), case["os"], case["oe"])
        torch.cuda.empty_cache()
        if kind == "medoid":
            return (None if d is None else d.cpu().numpy()), None, means, sigmas
        if d is None:
            return None
        n = case["n"]
        s, j = np.triu_indices(n, 1)
        sos = torch.zeros(n, dtype=torch.float64, device=d.device)
        sos.index_add_(0, torch.from_numpy(s).to(d.device), d * d)
        sos.index_add_(0, torch.from_numpy(j).to(d.device), d * d)
        return d, sos, None
    if kind == "round":
        return _exact_round(case, seed)
    if kind == "serve":
        reads, cents = _host_inputs(case, seed)
        reads, cents = _tensors(reads), _tensors(cents)
        d = _exact_dists([r for r in reads for _ in cents], [c for _ in reads for c in cents],
                         case["os"], case["oe"])
        torch.cuda.empty_cache()
        return None if d is None else d.cpu().numpy()
    # stripe rounds take longer than a plain restatement allows; segment
    # medians and whole averages select samples and paths by integer or rounded
    # rules, so they have no 64-bit value of their own
    return None
