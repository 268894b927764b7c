"""The work that users have this engine do, as cases that can be timed.

Sizes are those of the benchmark workloads (``fuel_gb300/workloads.py``,
``bench.py``) and generic smaller, larger and odd ones around them.  Host
arrays go through the Python classes, as a caller of ``fuel.search`` and
``fuel.cluster`` holds them; arrays that already live on the GPU go through
the C ABI, whose every pointer may be a device pointer.
"""
import ctypes
import math

import numpy as np
import torch

from fuel_gb300 import SearchIndex, _lib, kmeans
from fuel_gb300.serving import Server

DEV = "cuda"


def listed():
    return [
        # one user's lookup: a handful of rows against a small table, host arrays in and out
        {"name": "knn_lookup_host", "kind": "knn", "api": "host", "dtype": "f32", "data": "mixture", "n": 10007,
         "d": 17, "m": 3, "k": 5, "self": False, "metric": "euclidean"},
        # all-points neighbour lists of a small low-dimensional set (the input of LOF, OPTICS)
        {"name": "knn_selfjoin_16d", "kind": "knn", "api": "device", "dtype": "f32", "data": "mixture", "n": 20000,
         "d": 16, "m": 20000, "k": 10, "self": True, "metric": "sqeuclidean"},
        # the large self-join on count data with many ties
        {"name": "knn_selfjoin_128d", "kind": "knn", "api": "device", "dtype": "f32", "data": "geometric",
         "n": 1000000, "d": 128, "m": 1000000, "k": 100, "self": True, "metric": "sqeuclidean"},
        # a small batch of embedding queries against a large resident index
        {"name": "knn_few_96d", "kind": "knn", "api": "device", "dtype": "f32", "data": "unit", "n": 2000000,
         "d": 96, "m": 16, "k": 10, "self": False, "metric": "sqeuclidean"},
        # a burst of serving requests of mixed size and k against the same kind of index
        {"name": "serve_burst_96d", "kind": "serve", "n": 2000000, "d": 96, "requests": 24, "largest": 4096},
        # neighbourhoods within a radius (the input of DBSCAN)
        {"name": "range_selfjoin_16d", "kind": "range", "n": 20000, "d": 16, "m": 20000, "metric": "euclidean"},
        # numpy's default dtype: the float64 self-join
        {"name": "knn_selfjoin_f64", "kind": "knn", "api": "device", "dtype": "f64", "data": "mixture", "n": 20000,
         "d": 16, "m": 20000, "k": 10, "self": True, "metric": "euclidean"},
        # the condensed distance matrix (the input of hierarchical clustering), odd size
        {"name": "pairwise_condensed", "kind": "pairwise", "n": 20001, "d": 16, "form": "condensed",
         "metric": "euclidean"},
        # an analyst's small clustering, host arrays, run until it converges
        {"name": "kmeans_small_host", "kind": "kmeans", "api": "host", "data": "mixture", "n": 3000, "d": 10, "k": 8,
         "max_iter": 100, "fixed": False},
        # image-like data of 8-bit values: the headline workload
        {"name": "kmeans_784d", "kind": "kmeans", "api": "device", "data": "sparse", "n": 70000, "d": 784, "k": 64,
         "max_iter": 100, "fixed": True},
        # real-valued features of odd sizes, run until it converges
        {"name": "kmeans_100d", "kind": "kmeans", "api": "device", "data": "mixture", "n": 100003, "d": 100, "k": 37,
         "max_iter": 50, "fixed": False},
        # hundreds of independent problems of uneven size in one call
        {"name": "kmeans_batched_512", "kind": "batched", "count": 512, "max_iter": 20},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["knn", "knn", "knn", "knn64", "serve", "range", "pairwise", "kmeans_host", "kmeans", "kmeans",
                       "batched"])
    if kind == "knn":
        d, n, k = _log(rng, 2, 256), _log(rng, 1000, 1000000), _log(rng, 1, 100)
        m = max(1, min(_log(rng, 1, 20000), int(2e12 / (n * d))))
        data = rng.choice(["mixture", "unit", "geometric"] if d >= 32 else ["mixture", "unit"])
        return {"kind": "knn", "api": rng.choice(["host", "device", "device"]), "dtype": "f32", "data": data, "n": n,
                "d": d, "m": m, "k": k, "self": False, "metric": rng.choice(["euclidean", "sqeuclidean"])}
    if kind == "knn64":
        d, n = _log(rng, 2, 64), _log(rng, 500, 30000)
        m = max(1, min(_log(rng, 1, n), int(1e10 / (n * d))))
        return {"kind": "knn", "api": rng.choice(["host", "device"]), "dtype": "f64", "data": "mixture", "n": n,
                "d": d, "m": m, "k": _log(rng, 1, 50), "self": False,
                "metric": rng.choice(["euclidean", "sqeuclidean"])}
    if kind == "serve":
        return {"kind": "serve", "n": _log(rng, 100000, 2000000), "d": rng.randint(32, 128),
                "requests": rng.randint(4, 24), "largest": _log(rng, 64, 4096)}
    if kind == "range":
        n = _log(rng, 1000, 40000)
        return {"kind": "range", "n": n, "d": _log(rng, 2, 64), "m": _log(rng, 1, n),
                "metric": rng.choice(["euclidean", "sqeuclidean"])}
    if kind == "pairwise":
        return {"kind": "pairwise", "n": _log(rng, 100, 20000), "d": _log(rng, 2, 256),
                "form": rng.choice(["condensed", "square"]), "metric": rng.choice(["euclidean", "sqeuclidean"])}
    if kind == "kmeans_host":
        return {"kind": "kmeans", "api": "host", "data": "mixture", "n": _log(rng, 200, 15000),
                "d": rng.randint(2, 40), "k": rng.randint(2, 32), "max_iter": 100, "fixed": False}
    if kind == "kmeans":
        d = _log(rng, 16, 784)
        n = min(_log(rng, 20000, 200000), int(6e7 / d))
        data = rng.choice(["mixture", "sparse"])
        return {"kind": "kmeans", "api": "device", "data": data, "n": n, "d": d, "k": _log(rng, 4, 256),
                "max_iter": rng.randint(10, 50), "fixed": data == "sparse"}
    return {"kind": "batched", "count": _log(rng, 8, 256), "max_iter": rng.randint(5, 20)}


# ---- inputs ----------------------------------------------------------------


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _mixture(g, n, d, centres, box, sd, dtype=torch.float32, queries=0):
    """Equal-weight isotropic Gaussian mixture, centres uniform in [-box, box]^d;
    `queries` more rows of the same mixture come after the first n."""
    c = (torch.rand(centres, d, generator=g, device=DEV, dtype=torch.float64) * 2 - 1) * box
    t = n + queries
    comp = torch.randint(0, centres, (t,), generator=g, device=DEV)
    x = c[comp] + sd * torch.randn(t, d, generator=g, device=DEV, dtype=torch.float64)
    return x.to(dtype).contiguous()


def _unit(g, t, d):
    x = torch.randn(t, d, generator=g, device=DEV, dtype=torch.float32)
    return (x / x.norm(dim=1, keepdim=True)).contiguous()


def _geometric(g, t, d):
    """Counts: min(geometric(0.1) - 1, 255) as float32."""
    u = torch.rand(t, d, generator=g, device=DEV, dtype=torch.float32).clamp_(min=1e-30)
    return torch.floor(torch.log(u) / math.log(0.9)).clamp_(0, 255).contiguous()


def _sparse(g, t, d):
    """8-bit values over 255, 80% zeros."""
    v = torch.randint(1, 256, (t, d), generator=g, device=DEV, dtype=torch.int16)
    v[torch.rand(t, d, generator=g, device=DEV) < 0.8] = 0
    return (v.to(torch.float32) / 255.0).contiguous()


def _knn_rows(case, seed):
    """(index rows, query rows) of a neighbour search."""
    g, n, d = _gen(seed), case["n"], case["d"]
    q = 0 if case.get("self") else case["m"]
    if case["data"] == "unit":
        x = _unit(g, n + q, d)
    elif case["data"] == "geometric":
        x = _geometric(g, n + q, d)
    else:
        x = _mixture(g, n, d, 6, 5.0, 0.5, torch.float64 if case["dtype"] == "f64" else torch.float32, q)
    return (x[:n].contiguous(), x[n:].contiguous()) if q else (x, x)


def _radius(case):
    # a little below the typical distance within a component: some tens of hits a row
    r = 0.5 * math.sqrt(2 * case["d"]) * (1 - 1.6 / math.sqrt(2 * case["d"]))
    return r * r if case["metric"] == "sqeuclidean" else r


def _range_room(case):
    """Entries that the caller has room for: far more than are found."""
    return case["m"] * (8 + case["n"] // 32)


def _range_rows(case, seed):
    x = _mixture(_gen(seed), case["n"], case["d"], 6, 5.0, 0.5)
    return x, x[:case["m"]].contiguous()


def _serve_rows(case, seed):
    """Index rows and the requests: (query rows, k), sizes log-uniform, k of three kinds."""
    g = _gen(seed)
    x = _unit(g, case["n"], case["d"])
    r = np.random.default_rng(case["requests"] * 7919 + case["largest"])  # the sizes are the case's
    sizes = np.exp(r.uniform(0.0, math.log(case["largest"] + 1), case["requests"])).astype(int).clip(1, case["largest"])
    ks = r.choice([1, 10, 100], case["requests"])
    return x, [(_unit(g, int(m), case["d"]), int(k)) for m, k in zip(sizes, ks)]


def _kmeans_rows(case, seed):
    g, n, d, k = _gen(seed), case["n"], case["d"], case["k"]
    x = _sparse(g, n, d) if case["data"] == "sparse" else _mixture(g, n, d, k, 10.0, 1.0)
    rows = torch.randperm(n, generator=g, device=DEV)[:k]
    return x, x[rows].contiguous()


def _problems(case):
    """(n, d, k) of each problem of a batched call; the sizes are the case's."""
    r = np.random.default_rng(case["count"])
    got = []
    for _ in range(case["count"]):
        n = int(np.exp(r.uniform(np.log(1000), np.log(200000))))
        d = int(r.choice((2, 8, 32, 64)))
        got.append((n, d, int(np.exp(r.uniform(np.log(4), np.log(256))))))
    return got


def _batched_rows(case, seed):
    g = _gen(seed)
    got = []
    for n, d, k in _problems(case):
        x = _mixture(g, n, d, k, 10.0, 1.0)
        got.append((x, x[torch.randperm(n, generator=g, device=DEV)[:k]].contiguous()))
    return got


class _Index:
    """A device-resident index made from rows on the GPU (fuelg_index_create)."""

    def __init__(self, x, metric):
        self.lib = _lib.load()
        self.h = ctypes.c_void_p()
        torch.cuda.synchronize()
        make = self.lib.fuelg_index_create_f64 if x.dtype == torch.float64 else self.lib.fuelg_index_create
        _lib.check(make(_lib.ptr(x), x.shape[0], x.shape[1], _lib.METRIC[metric],
                        _lib.ORDER[_lib.default_order()], ctypes.byref(self.h)))

    def __del__(self):
        if self.h:
            self.lib.fuelg_index_destroy(self.h)


def prepare(case, seed):
    s = dict(case)
    kind = case["kind"]
    if kind == "knn":
        x, q = _knn_rows(case, seed)
        m, k = case["m"], case["k"]
        if case["api"] == "host":
            xh = x.cpu().numpy()
            s["index"] = SearchIndex(xh, distance=case["metric"])
            s["q"] = xh if case["self"] else q.cpu().numpy()
        else:
            s["index"] = _Index(x, case["metric"])
            s["q"] = None if case["self"] else q
            s["idx"] = torch.empty(m, k, dtype=torch.int64, device=DEV)
            s["dist"] = torch.empty(m, k, dtype=x.dtype, device=DEV)
    elif kind == "serve":
        x, requests = _serve_rows(case, seed)
        s["index"] = SearchIndex(x.cpu().numpy(), distance="sqeuclidean")
        s["server"] = Server(s["index"])
        s["requests"] = [(q.cpu().numpy(), k) for q, k in requests]
    elif kind == "range":
        x, q = _range_rows(case, seed)
        s["index"], s["q"], s["radius"] = _Index(x, case["metric"]), q, _radius(case)
        room = _range_room(case)
        s["idx"] = torch.zeros(room, dtype=torch.int64, device=DEV)
        s["dist"] = torch.zeros(room, device=DEV)
    elif kind == "pairwise":
        n = case["n"]
        s["x"] = _mixture(_gen(seed), n, case["d"], 6, 5.0, 0.5)
        s["out"] = torch.empty(n * (n - 1) // 2 if case["form"] == "condensed" else n * n, device=DEV)
    elif kind == "kmeans":
        x, c0 = _kmeans_rows(case, seed)
        if case["api"] == "host":
            s["x"], s["c0"] = x.cpu().numpy(), c0.cpu().numpy()
        else:
            s["x"], s["c0"], s["centres"] = x, c0, torch.empty_like(c0)
            s["labels"] = torch.empty(case["n"], dtype=torch.int64, device=DEV)
    else:
        rows = _batched_rows(case, seed)
        s["rows"] = rows
        # the batched call reads host or device arrays and writes host arrays
        s["centres"] = np.zeros(sum(c.numel() for _, c in rows), np.float32)
        s["labels"] = np.zeros(sum(x.shape[0] for x, _ in rows), np.int64)
        probs, c, t = [], 0, 0
        for x, c0 in rows:
            probs.append(_lib.KMeansProblem(x.data_ptr(), x.shape[0], x.shape[1], c0.shape[0], c0.data_ptr(),
                                            s["centres"].ctypes.data + 4 * c, s["labels"].ctypes.data + 8 * t, 0, 0,
                                            0.0))
            c, t = c + c0.numel(), t + x.shape[0]
        s["problems"] = (_lib.KMeansProblem * len(probs))(*probs)
    return s


# ---- one pass --------------------------------------------------------------


def _run_knn(s):
    if s["api"] == "host":
        return s["index"].knn(s["q"], s["k"], exclude_self=s["self"])
    ix = s["index"]
    mode = _lib.EXCLUDE_LINEAR if s["self"] else _lib.EXCLUDE_NONE
    q = None if s["q"] is None else _lib.ptr(s["q"])
    if s["dtype"] == "f64":
        _lib.check(ix.lib.fuelg_knn_f64(ix.h, q, s["m"], s["k"], mode, _lib.ptr(s["idx"]), _lib.ptr(s["dist"]), None))
    else:
        _lib.check(ix.lib.fuelg_knn(ix.h, q, s["m"], s["k"], mode, _lib.PRECISION["auto"], _lib.ptr(s["idx"]),
                                    _lib.ptr(s["dist"]), None))
    return s["idx"], s["dist"]


def _run_serve(s):
    waiting = [s["server"].submit(q, k) for q, k in s["requests"]]
    return [r.result() for r in waiting]


def _run_range(s):
    ix, m = s["index"], s["m"]
    res = ctypes.c_void_p()
    _lib.check(ix.lib.fuelg_range(ix.h, _lib.ptr(s["q"]), m, s["radius"], 1, ctypes.byref(res), None))
    total = ctypes.c_int64()
    _lib.check(ix.lib.fuelg_range_size(res, None, ctypes.byref(total)))
    idx, dist = s["idx"], s["dist"]
    if total.value > idx.shape[0]:
        idx, dist = torch.empty(total.value, dtype=torch.int64, device=DEV), torch.empty(total.value, device=DEV)
    off = torch.empty(m + 1, dtype=torch.int64, device=DEV)
    _lib.check(ix.lib.fuelg_range_copy(res, _lib.ptr(off), _lib.ptr(idx), _lib.ptr(dist)))
    ix.lib.fuelg_range_free(res)
    return off, idx, dist


def _run_pairwise(s):
    form = 0 if s["form"] == "condensed" else 1
    _lib.check(_lib.load().fuelg_pairwise(_lib.ptr(s["x"]), s["n"], s["d"], _lib.METRIC[s["metric"]],
                                          _lib.ORDER[_lib.default_order()], form, _lib.ptr(s["out"]), None))
    return s["out"]


def _run_kmeans(s):
    if s["api"] == "host":
        r = kmeans(s["x"], k=s["k"], variant="lloyd", init=s["c0"], max_iter=s["max_iter"], fixed_iters=s["fixed"])
        return r.centers, r.labels, r.n_iter, r.inertia
    iters, inertia = ctypes.c_int32(), ctypes.c_double()
    _lib.check(_lib.load().fuelg_kmeans_lloyd(
        _lib.ptr(s["x"]), s["n"], s["d"], s["k"], _lib.ptr(s["c0"]), s["max_iter"], 0.0, _lib.PRECISION["auto"],
        _lib.ORDER[_lib.default_order()], _lib.LLOYD_FIXED_ITERS if s["fixed"] else 0, _lib.ptr(s["centres"]),
        _lib.ptr(s["labels"]), ctypes.byref(iters), ctypes.byref(inertia), None))
    return s["centres"], s["labels"], iters.value, inertia.value


def _run_batched(s):
    p = s["problems"]
    _lib.check(_lib.load().fuelg_kmeans_batched(ctypes.cast(p, ctypes.c_void_p), len(p), s["max_iter"],
                                                _lib.ORDER[_lib.default_order()], _lib.PRECISION["auto"],
                                                _lib.LLOYD_FIXED_ITERS, None))
    return s["centres"], s["labels"], np.array([t.out_inertia for t in p])


def run(state):
    return {"knn": _run_knn, "serve": _run_serve, "range": _run_range, "pairwise": _run_pairwise,
            "kmeans": _run_kmeans, "batched": _run_batched}[state["kind"]](state)


# ---- what a pass cannot do without -----------------------------------------


def work(case):
    """Inputs read once, outputs written once; a squared distance of d
    coordinates as the 2 d operations of its contraction."""
    kind, n, d = case["kind"], case.get("n", 0), case.get("d", 0)
    if kind == "knn":
        w, m, k = 8 if case["dtype"] == "f64" else 4, case["m"], case["k"]
        rows = n if case["self"] else n + m
        return {"bytes": rows * d * w + m * k * (8 + w), "flops": 2 * m * n * d}
    if kind == "serve":
        r = np.random.default_rng(case["requests"] * 7919 + case["largest"])
        sizes = np.exp(r.uniform(0.0, math.log(case["largest"] + 1), case["requests"])).astype(int)
        sizes = sizes.clip(1, case["largest"])
        ks = r.choice([1, 10, 100], case["requests"])
        m = int(sizes.sum())
        return {"bytes": (n + m) * d * 4 + int((sizes * ks).sum()) * 12, "flops": 2 * m * n * d}
    if kind == "range":
        return {"bytes": n * d * 4 + case["m"] * 8, "flops": 2 * case["m"] * n * d}
    if kind == "pairwise":
        outs = n * (n - 1) // 2 if case["form"] == "condensed" else n * n
        return {"bytes": n * d * 4 + outs * 4, "flops": n * (n - 1) * d}
    if kind == "kmeans":
        # a run that stops by itself makes at least two passes
        passes = case["max_iter"] if case["fixed"] else 2
        return {"bytes": passes * n * d * 4 + n * 8, "flops": passes * 2 * n * case["k"] * d}
    probs = _problems(case)
    return {"bytes": sum(case["max_iter"] * n * d * 4 + n * 8 for n, d, k in probs),
            "flops": sum(case["max_iter"] * 2 * n * d * k for n, d, k in probs)}


# ---- the same in 64 bits ---------------------------------------------------


def _dist64(q, x):
    """Squared distances in 64 bits, by differences."""
    return torch.cdist(q, x, compute_mode="donot_use_mm_for_euclid_dist").square_()


def _topk64(q, x, k, exclude_self, metric):
    """[m, k] distances in 64 bits, ascending.  Excluding self drops the point
    itself from its k nearest, as the linear index does."""
    x = x.double()
    k_all = min(x.shape[0], k)
    step = max(1, int(2e9 / (8 * x.shape[0])))
    x2 = (x * x).sum(1)
    got = []
    for a in range(0, q.shape[0], step):
        b = q[a:a + step].double()
        wide = min(x.shape[0], k_all + 8)
        near = (x2[None, :] - 2.0 * (b @ x.T)).topk(wide, dim=1, largest=False).indices
        dd = (b[:, None, :] - x[near]).square_().sum(2)
        if exclude_self:
            dd[near == torch.arange(a, a + b.shape[0], device=DEV)[:, None]] = math.inf
        dd = dd.sort(dim=1).values
        got.append(torch.cat([dd[:, :k - 1], torch.full_like(dd[:, :1], math.inf)], 1) if exclude_self else dd[:, :k])
    out = torch.cat(got)
    if out.shape[1] < k:
        out = torch.cat([out, out.new_full((out.shape[0], k - out.shape[1]), math.inf)], 1)
    return out.sqrt_() if metric == "euclidean" else out


def _lloyd64(x, c0, max_iter, fixed):
    """(centres, inertia of the last pass) of Lloyd's iteration in 64 bits."""
    x, c = x.double(), c0.double()
    old = None
    for it in range(max_iter):
        lab = (c * c).sum(1)[None, :].sub(2.0 * (x @ c.T)).argmin(1)
        used = c
        if old is not None and torch.equal(lab, old) and not fixed:
            break
        if old is None or it + 1 < max_iter or fixed:
            one = torch.zeros_like(c).index_add_(0, lab, x)
            cnt = torch.bincount(lab, minlength=c.shape[0])
            c = torch.where(cnt[:, None] > 0, one / cnt.clamp(min=1)[:, None], c)
        old = lab
    return c, float((x - used[lab]).square_().sum())


def exact(case, seed):
    kind = case["kind"]
    if kind == "knn":
        if case["m"] * case["n"] * case["d"] > 5e12:  # minutes in 64 bits
            return None
        x, q = _knn_rows(case, seed)
        if case["api"] == "host":
            x, q = x.cpu().to(DEV), q.cpu().to(DEV)
        return None, _topk64(q, x, case["k"], case["self"], case["metric"])
    if kind == "serve":
        x, requests = _serve_rows(case, seed)
        x = x.double()
        return [(None, _topk64(q, x, k, False, "sqeuclidean")) for q, k in requests]
    if kind == "range":
        x, q = _range_rows(case, seed)
        x = x.double()
        r = _radius(case)
        rows, dist = [], []
        step = max(1, int(2e9 / (8 * case["n"])))
        for a in range(0, case["m"], step):
            dd = _dist64(q[a:a + step].double(), x)
            if case["metric"] == "euclidean":
                dd = dd.sqrt_()
            me = torch.arange(dd.shape[0], device=DEV)
            dd[me, me + a] = math.inf
            hit = (dd <= r).nonzero()
            rows.append(hit[:, 0] + a)
            dist.append(dd[hit[:, 0], hit[:, 1]])
        rows, dist = torch.cat(rows), torch.cat(dist)
        o = dist.argsort(stable=True)
        o = o[rows[o].argsort(stable=True)]
        out = torch.zeros(max(_range_room(case), dist.shape[0]), dtype=torch.float64, device=DEV)
        out[:dist.shape[0]] = dist[o]
        return None, None, out
    if kind == "pairwise":
        n = case["n"]
        x = _mixture(_gen(seed), n, case["d"], 6, 5.0, 0.5).double()
        out = torch.empty(n * (n - 1) // 2 if case["form"] == "condensed" else n * n, dtype=torch.float64, device=DEV)
        for a in range(0, n, 1024):
            dd = _dist64(x[a:a + 1024], x)
            if case["metric"] == "euclidean":
                dd = dd.sqrt_()
            if case["form"] == "square":
                out[a * n:a * n + dd.numel()] = dd.reshape(-1)
                continue
            i = torch.arange(a, a + dd.shape[0], device=DEV)[:, None]
            keep = torch.arange(n, device=DEV)[None, :] < i
            first = a * (a - 1) // 2
            low = dd[keep]
            out[first:first + low.numel()] = low
        return out
    if kind == "kmeans":
        if case["data"] == "sparse":
            return None  # no cluster structure: a rounding decides where the run goes
        x, c0 = _kmeans_rows(case, seed)
        c, inertia = _lloyd64(x, c0, case["max_iter"], case["fixed"])
        return c, None, None, inertia
    return None  # some problem of the batch always has points halfway between two centres
