"""What the engine is used for, as cases that can be timed and compared.

A case is a dict of plain values.  `prepare` makes what a caller holds before
the call (graphs built, queries and resident batches in place), `run` is one
pass through the package's public entry points, `work` is what the path cannot
do without, and `exact` is the same result in plain numpy float64.

Kinds of case, and who makes such calls:

* fit      one whole graph, from 30 edges to the 28M-edge power-law graph: the
           similarity of every edge.  A program that refits a graph resets the
           edge values (a fit goes on from the values it finds) and reads the
           edge and vertex values where the graph keeps them.
* delta,   fingerprints of graphs: the exact histogram over all vertex-deleted
  nabla    (vertex-marked) subgraphs; one small graph while a user waits,
           a list of graphs of mixed sizes, one strided share of a Delta^2
           that several workers divide between them, and a vertex-transitive
           graph (the graphs that fingerprints are asked to tell apart), whose
           histogram is short for the many values it counts.  The program
           collects the histograms in a table, a row a graph.
* batch    the same, resident on the device: run again and fetched.
* get      link prediction: the value that absent edges would have.
* hist     the histogram of values that are already on the device, for callers
           that cannot allocate.
* serve    a burst of mixed requests through the request server.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(ROOT, "dress-graph_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import dress_b200 as db  # noqa: E402
from dress_b200 import graphs  # noqa: E402

MAX_ITER, EPS = 100, 1e-6
#: Sweeps of a fit that `work` counts: about what epsilon 1e-6 takes.
SWEEPS = 20


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # the smallest request of a serving stream: latency and launches alone
        dict(name="fit regular 30 edges", kind="fit", model="regular", n=20, d=3, weighted=False, nw=False,
             variant=db.UNDIRECTED),
        # the plain fit of the benchmark: one Erdos-Renyi graph, G(2000, 10000)
        dict(name="fit G(2000,10000)", kind="fit", model="er", n=2000, m=10000, weighted=False, nw=False,
             variant=db.UNDIRECTED),
        # a large request of a serving stream: power law, weighted, odd sizes
        dict(name="fit power law 200k", kind="fit", model="chunglu", n=28573, m=200003, weighted=True, nw=False,
             variant=db.UNDIRECTED),
        # the large single fit of the benchmark: 4M vertices, 28M weighted edges
        dict(name="fit power law 28M", kind="fit", model="chunglu", n=4_000_000, m=28_000_000, weighted=True,
             nw=False, variant=db.UNDIRECTED),
        # one small graph's fingerprint, a user waiting
        dict(name="delta1 one graph", kind="delta", model="regular", count=1, n_lo=61, n_hi=61, d_lo=6, d_hi=6,
             k=1, stride=1, weighted=True),
        # a list of graphs of the benchmark's sizes (16..100 vertices, degree 3..12)
        dict(name="delta1 60 graphs", kind="delta", model="regular", count=60, n_lo=16, n_hi=100, d_lo=3, d_hi=12,
             k=1, stride=1, weighted=False),
        # one worker's share (1 of 64) of the benchmark's Delta^2: 10-regular
        # graphs of 200 vertices
        dict(name="delta2 share 8 graphs", kind="delta", model="regular", count=8, n_lo=200, n_hi=200, d_lo=10,
             d_hi=10, k=2, stride=64, weighted=False),
        # vertex-transitive graphs: many values, few of them distinct; the
        # first pair's Delta^2, and the Nabla^1 (the benchmark's sizes) of a
        # list that is resident on the device and run again
        dict(name="delta2 circulant pair", kind="delta", model="circulant", count=2, n_lo=101, n_hi=101, d_lo=10,
             d_hi=10, k=2, stride=1, weighted=False),
        dict(name="nabla1 batch 24 graphs", kind="batch", model="circulant", count=24, n_lo=200, n_hi=200, d_lo=10,
             d_hi=10, k=1, stride=1, weighted=False),
        # link prediction on a fitted power-law graph
        dict(name="get 100k pairs", kind="get", n=28573, m=200003, queries=100003),
        # a histogram without allocation, at the entry point's largest size
        dict(name="hist 1M values", kind="hist", values=1 << 20, distinct=1 << 19),
        # a burst of requests of a serving stream, 30 % of them Delta^1
        dict(name="serve 24 requests", kind="serve", count=24, fit_hi=100_000, delta_hi=1000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fit", "fit", "fit", "delta", "delta", "batch", "get", "hist", "serve"])
    weighted = rng.random() < 0.3
    if kind == "fit":
        m = _log_int(rng, 30, 3_000_000)
        if m < 5000 and rng.random() < 0.5:
            d = rng.randint(3, 12)
            n = max(d + 2, 2 * m // d)
            return dict(kind="fit", model="regular", n=n + (n * d) % 2, d=d, weighted=weighted,
                        nw=rng.random() < 0.2, variant=db.UNDIRECTED)
        if m < 30000:
            return dict(kind="fit", model="er", n=max(int(math.sqrt(4 * m)) + 2, m // rng.randint(3, 8)), m=m,
                        weighted=weighted, nw=rng.random() < 0.2,
                        variant=rng.choice([db.UNDIRECTED, db.UNDIRECTED, db.DIRECTED, db.FORWARD]))
        return dict(kind="fit", model="chunglu", n=max(16, m // 7), m=m, weighted=weighted, nw=rng.random() < 0.2,
                    variant=db.UNDIRECTED)
    if kind in ("delta", "batch"):
        n_lo = rng.randint(16, 150)
        n_hi = rng.randint(n_lo, 200)
        d_lo = rng.randint(3, 8)
        k = 2 if kind == "delta" and rng.random() < 0.4 else 1
        model = rng.choice(["regular", "regular", "circulant"])
        return dict(kind=kind, model=model, count=_log_int(rng, 1, 60 if n_hi < 120 else 12),
                    n_lo=n_lo, n_hi=n_hi, d_lo=d_lo, d_hi=rng.randint(d_lo, 12), k=k,
                    stride=rng.randint(48, 64) if k == 2 else 1, weighted=weighted)
    if kind == "get":
        m = _log_int(rng, 2000, 200_000)
        return dict(kind="get", n=max(16, m // 7), m=m, queries=_log_int(rng, 100, 100_000))
    if kind == "hist":
        v = _log_int(rng, 1000, 1 << 20)
        return dict(kind="hist", values=v, distinct=max(1, int(v * rng.random())))
    return dict(kind="serve", count=rng.randint(8, 24), fit_hi=_log_int(rng, 2000, 100_000),
                delta_hi=_log_int(rng, 100, 1000))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _power_law(n, m, seed, gamma=2.3):
    """The package's Chung-Lu model (graphs.chung_lu), drawn with torch on the
    GPU: that generator takes half a minute for 28M edges."""
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    cap = float(min(20000, n // 2))
    w = torch.arange(1, n + 1, dtype=torch.float64, device=dev) ** (-1.0 / (gamma - 1.0))
    w *= (2.0 * m / n) / w.mean()
    for _ in range(50):
        over = w > cap
        if not bool(over.any()):
            break
        w[over] = cap
        w[~over] *= (2.0 * m - float(w[over].sum())) / float(w[~over].sum())
    cdf = torch.cumsum(w, 0)
    cdf /= cdf[-1].clone()
    keys = torch.zeros(0, dtype=torch.int64, device=dev)
    while keys.numel() < m:
        need = int((m - keys.numel()) * 1.3) + 1024
        a = torch.searchsorted(cdf, torch.rand(need, dtype=torch.float64, device=dev, generator=gen)).clamp_(0, n - 1)
        b = torch.searchsorted(cdf, torch.rand(need, dtype=torch.float64, device=dev, generator=gen)).clamp_(0, n - 1)
        lo, hi = torch.minimum(a, b), torch.maximum(a, b)
        keep = lo != hi
        keys = torch.unique(torch.cat([keys, lo[keep] * n + hi[keep]]))
    keys = keys[torch.randperm(keys.numel(), device=dev, generator=gen)[:m]]
    perm = torch.randperm(n, device=dev, generator=gen)
    U = perm[keys // n].to(torch.int32).cpu().numpy()
    V = perm[keys % n].to(torch.int32).cpu().numpy()
    del w, cdf, keys, perm
    torch.cuda.empty_cache()
    return n, U, V


def _circulant(n, d, rng):
    """The circulant graph of d/2 random offsets, its vertices shuffled."""
    offs = rng.choice(np.arange(1, (n - 1) // 2 + 1), size=d // 2, replace=False)
    i = np.arange(n)
    U = np.concatenate([i for _ in offs])
    V = np.concatenate([(i + o) % n for o in offs])
    p = rng.permutation(n)
    return n, p[U].astype(np.int32), p[V].astype(np.int32)


def _model(case, seed):
    if case["model"] == "regular":
        return graphs.random_regular(case["n"], case["d"], seed=seed)
    if case["model"] == "er":
        return graphs.erdos_renyi(case["n"], case["m"], seed=seed)
    return _power_law(case["n"], case["m"], seed)


def _fit_inputs(case, seed):
    n, U, V = _model(case, seed)
    W = graphs.uniform_weights(len(U), seed=seed + 1) if case["weighted"] else None
    NW = graphs.uniform_weights(n, seed=seed + 2) if case["nw"] else None
    return n, U, V, W, NW


def _list_inputs(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(case["count"]):
        n = int(rng.integers(case["n_lo"], case["n_hi"] + 1))
        d = int(rng.integers(case["d_lo"], case["d_hi"] + 1))
        if case["model"] == "circulant":
            n, U, V = _circulant(n, d, rng)
        else:
            n, U, V = graphs.random_regular(n + (n * d) % 2, d, seed=int(rng.integers(1 << 31)))
        W = rng.uniform(0.5, 2.0, len(U)) if case["weighted"] else None
        out.append((n, U, V, W))
    return out


def _pairs(n, U, V, count, seed):
    """Half of the pairs random, half two steps apart (where links are sought)."""
    rng = np.random.default_rng(seed)
    off, tgt = _rows(n, U, V)[:2]
    u = rng.integers(0, n, count)
    v = rng.integers(0, n, count)
    near = rng.random(count) < 0.5
    e = rng.integers(0, len(U), count)
    mid, far = U[e], V[e]
    pick = off[far] + (rng.random(count) * (off[far + 1] - off[far])).astype(np.int64)
    u[near], v[near] = mid[near], tgt[pick][near]
    return u.astype(np.int32), v.astype(np.int32)


def _hist_values(case, seed):
    """Values as fits leave them: in (0, 1], each several times over."""
    rng = np.random.default_rng(seed)
    distinct = 0.05 + 0.95 * rng.random(case["distinct"]) ** 2
    return distinct[rng.integers(0, case["distinct"], case["values"])]


def _graph(n, U, V, W=None, NW=None, variant=db.UNDIRECTED):
    return db.Graph(n, U, V, W, NW, variant, device_build=len(U) >= 1_000_000)


class _Held:
    """n doubles of a graph's own memory; the graph lives as long as they do."""

    def __init__(self, g, ptr, n):
        self.g = g
        self.__array_interface__ = dict(shape=(n,), typestr="<f8", version=3,
                                        data=(ctypes.cast(ptr, ctypes.c_void_p).value, False))


def _edge_values(g):
    """The graph's own edge and vertex values, as tensors over its memory."""
    c = g.ptr.contents
    return (torch.from_numpy(np.asarray(_Held(g, c.edge_dress, g.E))),
            torch.from_numpy(np.asarray(_Held(g, c.vertex_dress, g.N))))


_server = None


def _the_server():
    global _server
    if _server is None:
        _server = db.Server()
    return _server


def prepare(case, seed):
    kind = case["kind"]
    if kind == "fit":
        g = _graph(*_fit_inputs(case, seed), case["variant"])
        e, v = _edge_values(g)
        return dict(kind=kind, g=g, edge=e, vertex=v)
    if kind in ("delta", "batch"):
        gs = [_graph(*x) for x in _list_inputs(case, seed)]
        opts = dict(k=case["k"], stride=case["stride"], offset=seed % case["stride"], max_iterations=MAX_ITER,
                    epsilon=EPS)
        table = _table(case["count"], _most_values(case))
        if kind == "batch":
            return dict(kind=kind, batch=db.Batch(gs, db.NABLA, **opts), **table)
        return dict(kind=kind, gs=gs, opts=opts, **table)
    if kind == "get":
        n, U, V = _power_law(case["n"], case["m"], seed)
        g = _graph(n, U, V)
        db.fit_graph(g, MAX_ITER, EPS)
        u, v = _pairs(n, U, V, case["queries"], seed + 1)
        return dict(kind=kind, g=g, u=u, v=v)
    if kind == "hist":
        vals = torch.from_numpy(_hist_values(case, seed)).cuda()
        return dict(kind=kind, vals=vals, pairs=torch.zeros(2 * vals.numel(), dtype=torch.int64, device="cuda"),
                    runs=torch.zeros(1, dtype=torch.int64, device="cuda"))
    reqs = []
    for what, n, U, V, W in _serve_inputs(case, seed):
        g = _graph(n, U, V, W)
        reqs.append((what, g) + _edge_values(g))
    hists = [g for what, g, _, _ in reqs if what == db.DELTA]
    return dict(kind=kind, server=_the_server(), reqs=reqs,
                **_table(len(hists), max([g.N * g.E for g in hists], default=1)))


def _most_values(case):
    """The values of one graph's subgraphs, at most."""
    n = case["n_hi"] + 1
    fits = n if case["k"] == 1 else n * (n - 1) // 2 // case["stride"] + 1
    return fits * (n * case["d_hi"] // 2)


def _table(count, most):
    table = torch.zeros((count, 2 * most), dtype=torch.int64)
    return dict(table=table, rows=list(table.numpy()), lens=torch.zeros(count, dtype=torch.int64))


def _enter(state, row, flat):
    state["rows"][row][:len(flat)] = flat
    state["lens"][row] = len(flat)


def _serve_inputs(case, seed):
    """Requests as in graphs.serving_stream: 30 % Delta^1, 30 % weighted, edge
    counts log-uniform, regular graphs below 5,000 edges and power laws above.
    The sizes are the case's, the graphs the seed's."""
    rng, out = np.random.default_rng(case["count"]), []
    for i in range(case["count"]):
        what = db.DELTA if i % 10 in (2, 5, 8) else db.FIT
        m = int(round(math.exp(rng.uniform(math.log(10), math.log(case["delta_hi"] if what == db.DELTA
                                                                   else case["fit_hi"])))))
        s = (seed * 1000 + i) % (1 << 31)
        if m < 5000:
            d = int(rng.integers(3, 13))
            n = max(2 * d, 2 * m // d)
            n, U, V = graphs.random_regular(n + (n * d) % 2, d, seed=s)
        else:
            n = m // 7
            n, U, V = graphs.chung_lu(n, m, 2.3, min(20000, n // 2), seed=s)
        W = graphs.uniform_weights(len(U), seed=s + 1) if rng.random() < 0.3 else None
        out.append((what, n, U, V, W))
    return out


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "fit":
        state["edge"].fill_(1.0)
        it, delta = db.fit_graph(state["g"], MAX_ITER, EPS)
        return dict(edge=state["edge"], vertex=state["vertex"], iterations=it, delta=delta)
    if kind == "delta":
        for i, flat in enumerate(db.delta_fit_many(state["gs"], **state["opts"])):
            _enter(state, i, flat)
        return dict(table=state["table"], lens=state["lens"])
    if kind == "batch":
        state["batch"].run()
        for i, flat in enumerate(state["batch"].fetch()):
            _enter(state, i, flat)
        return dict(table=state["table"], lens=state["lens"])
    if kind == "get":
        return db.get(state["g"], state["u"], state["v"], MAX_ITER, EPS)
    if kind == "hist":
        vals, pairs, runs = state["vals"], state["pairs"], state["runs"]
        rc = db.lib().dressx_histogram_noalloc(ctypes.c_void_p(vals.data_ptr()), vals.numel(),
                                               ctypes.c_void_p(pairs.data_ptr()), ctypes.c_void_p(runs.data_ptr()),
                                               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise db.DressError(rc, "dressx_histogram_noalloc")
        return dict(pairs=pairs, runs=runs)
    tickets = []
    for what, g, edge, vertex in state["reqs"]:
        if what == db.FIT:
            edge.fill_(1.0)
        tickets.append(state["server"].submit(g, what, 0 if what == db.FIT else 1, MAX_ITER, EPS))
    fits, row = [], 0
    for (what, g, edge, vertex), t in zip(state["reqs"], tickets):
        r = t.wait()
        if r["status"]:
            raise db.DressError(r["status"], "served request")
        if what == db.FIT:
            fits.append([edge, vertex])
        else:
            _enter(state, row, r["hist_flat"])
            row += 1
    return dict(fits=fits, table=state["table"], lens=state["lens"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def _fit_work(n, E, slots):
    """One fit: the rows, the endpoints, weights and values in, the values
    out; a product and a sum a slot, the update of an edge, a sweep."""
    return dict(bytes=4 * (n + 1) + 8 * slots + 24 * E + 8 * E + 8 * n, flops=SWEEPS * (2 * slots + 6 * E))


def work(case):
    kind = case["kind"]
    if kind == "fit":
        E = case["n"] * case["d"] // 2 if case["model"] == "regular" else case["m"]
        return _fit_work(case["n"], E, (1 if case["variant"] == db.FORWARD else 2) * E)
    if kind in ("delta", "batch"):
        n, d = (case["n_lo"] + case["n_hi"]) / 2, (case["d_lo"] + case["d_hi"]) / 2
        E = n * d / 2
        fits = case["count"] * (n if case["k"] == 1 else n * (n - 1) / 2) / case["stride"]
        # at most a (value, count) pair for each value; a vertex-transitive
        # graph's n subsets of an orbit share theirs
        pairs = fits * E / (n if case["model"] == "circulant" else 1)
        return dict(bytes=case["count"] * _fit_work(n, E, 2 * E)["bytes"] + 16 * pairs,
                    flops=fits * _fit_work(n, E, 2 * E)["flops"])
    if kind == "get":
        E, q = case["m"], case["queries"]
        return dict(bytes=4 * (case["n"] + 1) + 16 * E + 16 * E + 8 * case["n"] + 16 * q,
                    flops=q * (20 * 8 + 4 * E / case["n"]))
    if kind == "hist":
        distinct = case["distinct"] * (1 - math.exp(-case["values"] / case["distinct"]))
        return dict(bytes=8 * case["values"] + 16 * distinct, flops=0)
    fits, deltas = 0.7 * case["count"], 0.3 * case["count"]
    ef = case["fit_hi"] / math.log(case["fit_hi"] / 10)
    ed = case["delta_hi"] / math.log(case["delta_hi"] / 10)
    f, d = _fit_work(ef / 7, ef, 2 * ef), _fit_work(ed / 4, ed, 2 * ed)
    return dict(bytes=fits * f["bytes"] + deltas * (d["bytes"] + 16 * ed * ed / 4),
                flops=fits * f["flops"] + deltas * ed / 4 * d["flops"])


# ---------------------------------------------------------------------------
# the same results in plain float64
# ---------------------------------------------------------------------------

def _rows(n, U, V, variant=db.UNDIRECTED):
    """off, targets, edge ids of the rows, ascending by target."""
    e = np.arange(len(U))
    if variant == db.FORWARD:
        r, t, i = U, V, e
    else:
        r, t, i = np.concatenate([U, V]), np.concatenate([V, U]), np.concatenate([e, e])
    order = np.lexsort((t, r))
    off = np.zeros(n + 1, dtype=np.int64)
    np.cumsum(np.bincount(r, minlength=n), out=off[1:])
    return off, t[order].astype(np.int64), i[order]


def _common(n, off, tgt, eid, a, b):
    """(query, edge (a,x), edge (b,x)) of every common neighbour x of each (a, b)."""
    deg = off[1:] - off[:-1]
    swap = deg[a] > deg[b]
    s, l = np.where(swap, b, a).astype(np.int64), np.where(swap, a, b).astype(np.int64)
    cnt = deg[s]
    q = np.repeat(np.arange(len(a)), cnt)
    slot = np.arange(int(cnt.sum())) - np.repeat(np.cumsum(cnt) - cnt, cnt) + np.repeat(off[s], cnt)
    keys = np.repeat(np.arange(n), deg) * n + tgt
    want = l[q] * n + tgt[slot]
    at = np.minimum(np.searchsorted(keys, want), max(0, len(keys) - 1))
    hit = keys[at] == want if len(keys) else np.zeros(0, dtype=bool)
    return q[hit], eid[slot[hit]], eid[at[hit]]


def _fit_exact(n, U, V, W, NW, variant):
    E = len(U)
    w = (np.ones(E) if W is None else W) * (2.0 if variant == db.UNDIRECTED else 1.0)
    nw = np.ones(n) if NW is None else NW
    off, tgt, eid = _rows(n, U, V, variant)
    row = np.repeat(np.arange(n), off[1:] - off[:-1])
    pe, px, py = _common(n, off, tgt, eid, U, V)
    d = np.ones(E)
    it, delta = 0, 0.0
    for it in range(MAX_ITER):
        p = w * d
        vd = np.sqrt(4.0 * nw + np.bincount(row, p[eid], minlength=n))
        num = 4.0 * nw[U] + (p if variant == db.FORWARD else 4.0 * nw[V] + 2.0 * p)
        num = num + np.bincount(pe, p[px] + p[py], minlength=E)
        new = num / (vd[U] * vd[V])
        delta = float(np.max(np.abs(new - d)))
        d = new
        if delta < EPS:
            break
    else:
        it = MAX_ITER
    return d, vd, it, delta


def exact(case, seed):
    kind = case["kind"]
    if kind == "fit":
        if case.get("m", 0) > 1_000_000:
            return None                    # minutes of plain numpy
        e, v, it, delta = _fit_exact(*_fit_inputs(case, seed), case["variant"])
        return dict(edge=e, vertex=v, iterations=it, delta=delta)
    if kind == "get":
        n, U, V = _power_law(case["n"], case["m"], seed)
        d, vd, _, _ = _fit_exact(n, U, V, None, None, db.UNDIRECTED)
        u, v = _pairs(n, U, V, case["queries"], seed + 1)
        off, tgt, eid = _rows(n, U, V)
        q, ex, ey = _common(n, off, tgt, eid, u, v)
        a = 8.0 + np.bincount(q, 2.0 * d[ex] + 2.0 * d[ey], minlength=len(u))
        x = np.ones(len(u))
        live = np.ones(len(u), dtype=bool)
        for _ in range(MAX_ITER):
            nx = (a + 4.0 * x) / (np.sqrt(vd[u] ** 2 + 2.0 * x) * np.sqrt(vd[v] ** 2 + 2.0 * x))
            stop = np.abs(nx - x) <= EPS
            x = np.where(live, nx, x)
            live &= ~stop
        deg = off[1:] - off[:-1]
        keys = np.repeat(np.arange(n), deg) * n + tgt
        want = u.astype(np.int64) * n + v
        at = np.minimum(np.searchsorted(keys, want), len(keys) - 1)
        return np.where(keys[at] == want, d[eid[at]], x)
    if kind == "serve":
        return dict(fits=[list(_fit_exact(n, U, V, W, None, db.UNDIRECTED)[:2])
                          for what, n, U, V, W in _serve_inputs(case, seed) if what == db.FIT])
    return None                            # histograms are whole numbers: value bits and counts
