"""The batch kernel at the sizes and values where its paths change, bit for bit
against the oracle: edge counts around a warp and a word of live bits, weights
that are one power of two, one other value and mixed, products outside the
range of its short sums, marked and deleted vertices, and the forms of a
subgraph's state (products in shared memory, products formed per term, the
parent read through L2)."""
import numpy as np
import pytest

import dress_b200 as db
from dress_b200 import graphs

pytestmark = pytest.mark.gpu


def _weights(kind, m, rng):
    if kind == "none":
        return None
    return {"one": np.ones(m), "quarter": np.full(m, 0.25), "third": np.full(m, 0.3),
            "uniform": rng.uniform(0.5, 2.0, m), "heavy": rng.uniform(1.0, 400.0, m),
            "tiny": rng.uniform(1e-13, 1e-11, m), "zeros": rng.integers(0, 2, m).astype(float)}[kind]


def _sparse(n, m, seed):
    """A graph with isolated vertices, isolated edges and a few triangles."""
    assert m <= n * (n - 1) // 4
    rng = np.random.default_rng(seed)
    key = set()
    while len(key) < m:
        a, b = sorted(rng.integers(0, n, 2).tolist())
        if a != b:
            key.add((a, b))
    u, v = np.array(sorted(key)).T
    return n, u.astype(np.int32), v.astype(np.int32)


def _same(g, case, oracle_port, kind, k, **kw):
    n, U, V, W, variant = case
    ref_fn = oracle_port.delta_fit if kind == db.DELTA else oracle_port.nabla_fit
    ref = ref_fn(n, U, V, W, k=k, variant=variant, **kw)
    flat = db.hist_requests([g], kind, k, **kw)[0][0]
    np.testing.assert_array_equal(flat, ref["hist"])


@pytest.mark.parametrize("weights", ["none", "one", "quarter", "third", "uniform", "heavy", "tiny", "zeros"])
@pytest.mark.parametrize("m", [1, 2, 31, 32, 33, 63, 64, 65, 200])
def test_delta_and_nabla_of_sparse_graphs(m, weights, oracle_port):
    rng = np.random.default_rng(m)
    variant = [db.UNDIRECTED, db.DIRECTED, db.FORWARD, db.BACKWARD][m % 4]
    n, U, V = _sparse(max(4, int(1.2 * m) + 1) if m < 64 else 40, m, m)
    W = _weights(weights, m, rng)
    case = (n, U, V, W, variant)
    with db.Graph(n, U, V, W, variant=variant) as g:
        _same(g, case, oracle_port, db.DELTA, 1)
        _same(g, case, oracle_port, db.NABLA, 1)
        _same(g, case, oracle_port, db.DELTA, 2, n_samples=25, seed=m)
        _same(g, case, oracle_port, db.NABLA, 2, n_samples=25, seed=m)


@pytest.mark.parametrize("k", [1, 2, 3])
def test_every_rank_is_unranked(k, oracle_port):
    """All subsets and tuples of a graph with distinguishable vertices, and the
    multiset rows in the caller's edge order."""
    n, U, V = _sparse(40 if k < 3 else 14, 70 if k < 3 else 30, 5)
    with db.Graph(n, U, V) as g:
        for kind, fn in ((db.DELTA, oracle_port.delta_fit), (db.NABLA, oracle_port.nabla_fit)):
            ref = fn(n, U, V, k=k, keep_multisets=True)
            flat, ms = db.hist_requests([g], kind, k, keep_multisets=True)[0][:2]
            np.testing.assert_array_equal(flat, ref["hist"])
            np.testing.assert_array_equal(ms.view(np.int64), ref["multisets"].view(np.int64))


@pytest.mark.parametrize("n,m,weights", [(3000, 9000, "uniform"),      # products beside the values, one subgraph an SM
                                         (3000, 9800, "uniform"),      # products formed per term
                                         (2000, 12000, "none"),
                                         (150, 11175, "none"),         # complete: pairs read through L2
                                         (110, 5995, "uniform")])
def test_large_states(n, m, weights, oracle_port):
    n, U, V = graphs.erdos_renyi(n, m, seed=3)
    W = _weights(weights, m, np.random.default_rng(1))
    with db.Graph(n, U, V, W) as g:
        _same(g, (n, U, V, W, db.UNDIRECTED), oracle_port, db.DELTA, 1, n_samples=2, seed=4)


@pytest.mark.parametrize("m,weights,nw", [(1, "none", False), (32, "third", True), (33, "uniform", True),
                                          (700, "heavy", False), (1500, "none", True), (2048, "uniform", False)])
def test_plain_fits_in_one_cta(m, weights, nw, oracle_port):
    rng = np.random.default_rng(m)
    n, U, V = _sparse(max(14, m // 3), m, m)
    W = _weights(weights, m, rng)
    NW = rng.uniform(0.5, 3.0, n) if nw else None
    ref = oracle_port.fit(n, U, V, W, NW)
    with db.Graph(n, U, V, W, NW) as g:
        it, delta = db.fit_graph(g)
        assert (it, delta) == (ref["iterations"], ref["delta"])
        np.testing.assert_array_equal(g.edge_dress.view(np.int64), ref["edge_dress"].view(np.int64))
        np.testing.assert_array_equal(g.vertex_dress.view(np.int64), ref["vertex_dress"].view(np.int64))


def test_a_batch_of_every_size(oracle_port):
    """One launch over graphs of 1 to 2,000 edges: the states of one CTA's
    chunks differ in size and form."""
    rng = np.random.default_rng(8)
    cases = []
    for i, m in enumerate([1, 5, 40, 2000, 33, 700, 64, 1200, 2, 300]):
        n, U, V = _sparse(max(20, m // 4), m, i)
        cases.append((n, U, V, _weights(["none", "uniform", "heavy"][i % 3], m, rng)))
    gs = [db.Graph(*c) for c in cases]
    for kind, fn in ((db.DELTA, oracle_port.delta_fit), (db.NABLA, oracle_port.nabla_fit)):
        got = db.hist_requests(gs, kind, 1, n_samples=12, seed=2)
        for c, r in zip(cases, got):
            np.testing.assert_array_equal(r[0], fn(*c, k=1, n_samples=12, seed=2)["hist"])
    for g in gs:
        g.close()


@pytest.mark.parametrize("m,stride", [(20, 1), (33, 1), (200, 1), (1500, 40)])
def test_no_sweeps(m, stride, oracle_port):
    """max_iterations = 0: every live edge keeps its first value.  Groups of one
    and of several warps, repeated so that warps of a group meet in any order."""
    n, U, V = _sparse(max(14, m // 3), m, m)
    W = np.random.default_rng(m).uniform(0.5, 2.0, m)
    with db.Graph(n, U, V, W) as g:
        for kind, fn in ((db.DELTA, oracle_port.delta_fit), (db.NABLA, oracle_port.nabla_fit)):
            ref = fn(n, U, V, W, k=1, max_iterations=0, stride=stride)
            for _ in range(5):
                flat, _, _, fits, _ = db.hist_requests([g], kind, 1, max_iterations=0, stride=stride)[0]
                np.testing.assert_array_equal(flat, ref["hist"])
                assert flat.size and fits <= n
        with db.Server() as srv:
            r = srv.submit(g, db.DELTA, 1, max_iterations=0).wait()
            np.testing.assert_array_equal(r["hist_flat"], oracle_port.delta_fit(n, U, V, W, k=1, max_iterations=0)["hist"])


@pytest.mark.parametrize("weights", ["one to ten", "below four", "four", "one of five", "thousands", "growing"])
@pytest.mark.parametrize("n,m", [(14, 31), (40, 200), (110, 5995), (3000, 9800)])
def test_products_above_the_sums(n, m, weights, oracle_port):
    """Products that the four-addition sums do not take: at the edge of their
    range, far above it, in one edge only, and growing past it sweep by sweep,
    for every form of a subgraph's state."""
    rng = np.random.default_rng(m)
    n, U, V = graphs.erdos_renyi(n, m, seed=m)
    W = {"one to ten": rng.integers(1, 11, m).astype(float), "below four": rng.uniform(3.9, 4.0, m),
         "four": np.full(m, 4.0), "one of five": np.where(np.arange(m) == m // 2, 5.0, rng.uniform(0.5, 2.0, m)),
         "thousands": rng.uniform(1.0, 5000.0, m), "growing": np.exp(rng.uniform(-4.0, 2.0, m))}[weights]
    variant = [db.UNDIRECTED, db.FORWARD, db.BACKWARD][m % 3] if weights != "growing" else db.FORWARD
    with db.Graph(n, U, V, W, variant=variant) as g:
        _same(g, (n, U, V, W, variant), oracle_port, db.DELTA, 1, n_samples=4, seed=1)
        _same(g, (n, U, V, W, variant), oracle_port, db.NABLA, 1, n_samples=4, seed=2)


@pytest.mark.parametrize("m", [31, 300, 1023, 1024])
@pytest.mark.parametrize("lo,hi", [(0.05, 0.1), (0.2, 1.0), (0.6, 40.0), (1e-4, 1.0)])
def test_plain_fits_with_vertex_weights(m, lo, hi, oracle_port):
    """Vertex weights below 1 and far apart, up to the most edges of one CTA; a
    fit that goes on from values of its own."""
    rng = np.random.default_rng(m)
    n, U, V = _sparse(max(14, m // 3), m, m)
    W = rng.uniform(0.5, 2.0, m) if m % 2 else None
    NW = rng.uniform(lo, hi, n)
    ref = oracle_port.fit(n, U, V, W, NW)
    with db.Graph(n, U, V, W, NW) as g:
        db.counters(reset=True)
        db.fit_graph(g, 3, 0.0)
        it, delta = db.fit_graph(g)
        assert db.counters()["launches"] == 2
        assert (it + 3, delta) == (ref["iterations"], ref["delta"])
        np.testing.assert_array_equal(g.edge_dress.view(np.int64), ref["edge_dress"].view(np.int64))
        np.testing.assert_array_equal(g.vertex_dress.view(np.int64), ref["vertex_dress"].view(np.int64))
