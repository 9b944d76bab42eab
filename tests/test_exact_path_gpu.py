"""The sorted path behind the certified sums, on the GPU.

Every sum of the engine is a certified sum in gathering order; an item whose
certificate fails is summed the reference's way (sort ascending, then
sequential KBN, libdress/src/dress.c:51-66).  Real inputs almost never fail
the certificate, so these tests configure the engine with exact_sums=1,
which sends EVERY item down that sorted path, and require the same bits as
the oracle: the single-graph fit (shared-memory sorts and, for a hub beyond
shared memory, the global-scratch sort), the one-launch fits and the
batched Delta/Nabla kernel (its in-place selection order).
"""
import ctypes

import numpy as np
import pytest

import dress_b200 as db
from dress_b200 import graphs

pytestmark = pytest.mark.gpu


def bits(a):
    return np.asarray(a, dtype=np.float64).view(np.int64)


@pytest.fixture
def exact_sums():
    db.configure(exact_sums=1)
    try:
        yield
    finally:
        db.configure()


def gpu_fit(n, U, V, W=None, NW=None, variant=0, max_iterations=100, epsilon=1e-6):
    with db.Graph(n, U, V, W, NW, variant, 0) as g:
        it, dl = db.fit_graph(g, max_iterations, epsilon)
        return dict(edge_dress=g.edge_dress, vertex_dress=g.vertex_dress, iterations=it, delta=dl)


def assert_same(a, b):
    assert a["iterations"] == b["iterations"]
    assert bits([a["delta"]])[0] == bits([b["delta"]])[0]
    np.testing.assert_array_equal(bits(a["edge_dress"]), bits(b["edge_dress"]))
    np.testing.assert_array_equal(bits(a["vertex_dress"]), bits(b["vertex_dress"]))


def test_single_fit_sorted_path(oracle_port, exact_sums):
    # thread, warp and block items of a power-law graph, weighted, vertex weights
    n, U, V = graphs.chung_lu(20000, 120000, 2.3, 3000, seed=3)
    W = graphs.uniform_weights(len(U), seed=2)
    NW = np.random.default_rng(1).uniform(0.5, 2.0, n)
    assert_same(gpu_fit(n, U, V, W, NW, max_iterations=12), oracle_port.fit(n, U, V, W, NW, max_iterations=12))
    for variant in (1, 2):
        nn, U2, V2 = graphs.erdos_renyi(3000, 12000, seed=variant)
        assert_same(gpu_fit(nn, U2, V2, variant=variant), oracle_port.fit(nn, U2, V2, variant=variant))


def test_hub_beyond_shared_memory_sorted_path(oracle_port, exact_sums):
    # a 40000-leaf star: the hub's 40001 terms are sorted in global scratch
    n = 40001
    U = np.zeros(40000, np.int32)
    V = np.arange(1, 40001, dtype=np.int32)
    assert_same(gpu_fit(n, U, V, max_iterations=5), oracle_port.fit(n, U, V, max_iterations=5))


def test_one_launch_fits_sorted_path(oracle_port, exact_sums):
    for n, m in ((300, 1200), (1500, 6000)):
        n, U, V = graphs.erdos_renyi(n, m, seed=9)
        W = graphs.uniform_weights(m, seed=5)
        assert_same(gpu_fit(n, U, V, W), oracle_port.fit(n, U, V, W))


def test_batched_delta_nabla_sorted_path(oracle_port, exact_sums):
    gs = graphs.regular_batch(12, (16, 40), (3, 9), seed=4)
    objs = [db.Graph(n, U, V) for n, U, V in gs]
    for kind, fn in ((db.DELTA, oracle_port.delta_fit), (db.NABLA, oracle_port.nabla_fit)):
        flats = [r[0] for r in db.hist_requests(objs, kind, 1)]
        for (n, U, V), flat in zip(gs, flats):
            np.testing.assert_array_equal(flat, fn(n, U, V, k=1)["hist"])
    for g in objs:
        g.close()


def test_large_graph_layout_sorted_path(oracle_port, exact_sums):
    # the renumbered layout of a graph above 2^20 edges, every item sorted
    n, U, V = graphs.chung_lu(200_000, 1_200_000, 2.3, 3000, seed=5)
    W = graphs.uniform_weights(len(U), seed=6)
    assert_same(gpu_fit(n, U, V, W, max_iterations=4), oracle_port.fit(n, U, V, W, precompute=1, max_iterations=4))


@pytest.mark.parametrize("n,m", [(30, 100), (60, 900), (5000, 30001)])
def test_zero_weights_among_others(n, m, oracle_port):
    """Zero terms in most sums, of which many are ties between two doubles."""
    n, U, V = graphs.erdos_renyi(n, m, seed=m)
    W = np.random.default_rng(m).integers(0, 4, m).astype(float)
    W[::5] = -0.0
    ref = oracle_port.fit(n, U, V, W)
    with db.Graph(n, U, V, W) as g:
        it, delta = db.fit_graph(g)
        assert (it, delta) == (ref["iterations"], ref["delta"])
        np.testing.assert_array_equal(g.edge_dress.view(np.int64), ref["edge_dress"].view(np.int64))
        np.testing.assert_array_equal(g.vertex_dress.view(np.int64), ref["vertex_dress"].view(np.int64))


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan, 1e300, 5e-324])
@pytest.mark.parametrize("m", [100, 900, 3000, 30_001])
def test_weights_without_a_finite_sum(m, bad, oracle_port):
    """A NaN term, which sorts nowhere, makes its sum NaN on every path: one CTA,
    cluster, multi-kernel and the subgraphs of a batch."""
    n, U, V = graphs.erdos_renyi(max(30, m // 5), m, seed=m)
    W = np.random.default_rng(1).uniform(0.5, 2.0, m)
    W[[3, m // 2]] = bad
    ref = oracle_port.fit(n, U, V, W)
    with db.Graph(n, U, V, W) as g:
        it, delta = db.fit_graph(g)
        assert (it, delta) == (ref["iterations"], ref["delta"])
        np.testing.assert_array_equal(bits(g.edge_dress), bits(ref["edge_dress"]))
        np.testing.assert_array_equal(bits(g.vertex_dress), bits(ref["vertex_dress"]))
    if m < 1000 and not np.isnan(bad):
        with db.Graph(n, U, V, W) as g:
            flat = db.hist_requests([g], db.DELTA, 1, n_samples=8, seed=1)[0][0]
        np.testing.assert_array_equal(flat, oracle_port.delta_fit(n, U, V, W, k=1, n_samples=8, seed=1)["hist"])


@pytest.mark.parametrize("exact", [0, 1])
@pytest.mark.parametrize("pairs", [1, 40, 600, 30_000, 70_001])
def test_own_tables_longer_than_the_rows(pairs, exact, oracle_port):
    """A caller's tables may list more pairs for an edge than any row has slots:
    up to and beyond what a block sorts in shared memory."""
    n = 40
    U, V = np.arange(n - 1, dtype=np.int32), np.arange(1, n, dtype=np.int32)
    rng = np.random.default_rng(pairs)
    W = rng.uniform(0.5, 2.0, n - 1)
    off = np.zeros(n, np.int32)
    off[8:] = pairs                                  # all of them edge 7's
    ux, vx = (rng.integers(0, n - 1, pairs).astype(np.int32) for _ in range(2))
    names = ("intercept_offset", "intercept_edge_ux", "intercept_edge_vx")
    ip = ctypes.POINTER(ctypes.c_int)

    def fitted(c, fit):
        kept = [ctypes.cast(getattr(c, f), ctypes.c_void_p).value for f in names]
        c.max_degree = max(2, pairs)                 # what the oracle's buffer is sized by
        for f, a in zip(names, (off, ux, vx)):
            setattr(c, f, a.ctypes.data_as(ip))
        r = fit()
        for f, p in zip(names, kept):
            setattr(c, f, ctypes.cast(p, ip))
        return r, [np.ctypeslib.as_array(getattr(c, f), shape=(k,)).copy()
                   for f, k in (("edge_dress", n - 1), ("vertex_dress", n))]

    ref = oracle_port.build(n, U, V, W, None, db.UNDIRECTED, 1)
    it, delta = ctypes.c_int(), ctypes.c_double()
    _, want = fitted(ref.contents, lambda: oracle_port.fit_fn(ref, 20, 1e-6, ctypes.byref(it), ctypes.byref(delta)))
    oracle_port.free_graph(ref)
    db.configure(exact_sums=exact)
    try:
        with db.Graph(n, U, V, W, precompute_intercepts=True) as g:
            got, values = fitted(g.ptr.contents, lambda: db.fit_graph(g, 20))
    finally:
        db.configure()
    assert got == (it.value, delta.value)
    for a, b in zip(values, want):
        np.testing.assert_array_equal(bits(a), bits(b))
