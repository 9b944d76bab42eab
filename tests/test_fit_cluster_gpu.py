"""The one-launch cluster fit at the sizes and values where it changes shape,
bit for bit against the oracle: one and two value buffers, one to eight lanes a
vertex, edges a thread owns one to four of, variants, vertex weights, values to
go on from, and weights that take the fit off this path."""
import ctypes

import numpy as np
import pytest

import dress_b200 as db
from dress_b200 import graphs

pytestmark = pytest.mark.gpu


def _fit(oracle_port, n, U, V, W=None, NW=None, variant=db.UNDIRECTED, one_launch=True, **kw):
    ref = oracle_port.fit(n, U, V, W, NW, variant=variant, **kw)
    with db.Graph(n, U, V, W, NW, variant) as g:
        db.counters(reset=True)
        it, delta = db.fit_graph(g, kw.get("max_iterations", 100), kw.get("epsilon", 1e-6))
        launches = db.counters()["launches"]
        assert one_launch is None or (launches == 1) == one_launch
        assert (it, delta) == (ref["iterations"], ref["delta"])
        np.testing.assert_array_equal(g.edge_dress.view(np.int64), ref["edge_dress"].view(np.int64))
        np.testing.assert_array_equal(g.vertex_dress.view(np.int64), ref["vertex_dress"].view(np.int64))


@pytest.mark.parametrize("n,m", [(700, 2049), (2000, 8191), (2000, 8193), (2000, 10000), (120, 4000), (2600, 13000),
                                 (2700, 13300), (9000, 16385), (4000, 20000), (3600, 24576), (400, 24001),
                                 (8000, 22000), (16000, 24575), (500, 1025), (60000, 1500)])
def test_sizes(n, m, oracle_port):
    n, U, V = graphs.erdos_renyi(n, m, seed=m)
    rng = np.random.default_rng(m)
    W = rng.uniform(0.5, 2.0, m) if m % 2 else None
    _fit(oracle_port, n, U, V, W)


@pytest.mark.parametrize("variant", [db.UNDIRECTED, db.DIRECTED, db.FORWARD, db.BACKWARD])
@pytest.mark.parametrize("weights", ["none", "third", "wide"])
def test_variants_and_weights(variant, weights, oracle_port):
    n, U, V = graphs.erdos_renyi(900, 5003, seed=7)
    rng = np.random.default_rng(variant)
    W = {"none": None, "third": np.full(5003, 0.3), "wide": np.exp(rng.uniform(-6, 6, 5003))}[weights]
    NW = rng.uniform(0.3, 5.0, n) if weights != "none" else None
    # products over 37 binades and growing (FORWARD, BACKWARD) leave the range
    _fit(oracle_port, n, U, V, W, NW, variant, one_launch=None if weights == "wide" else True)


def test_multigraph_and_isolated_parts(oracle_port):
    """Parallel edges, self loops, isolated vertices and edges."""
    rng = np.random.default_rng(3)
    U = rng.integers(0, 800, 4000).astype(np.int32)
    V = rng.integers(0, 800, 4000).astype(np.int32)
    U[:50], V[:50] = np.arange(1000, 1050), np.arange(1050, 1100)
    _fit(oracle_port, 1200, U, V)


@pytest.mark.parametrize("iterations", [1, 2, 3, 7])
def test_few_sweeps_and_going_on(iterations, oracle_port):
    n, U, V = graphs.erdos_renyi(1000, 6000, seed=9)
    _fit(oracle_port, n, U, V, max_iterations=iterations)
    _fit(oracle_port, n, U, V, max_iterations=iterations, epsilon=0.0)
    # a second call goes on from the first one's values
    full = oracle_port.fit(n, U, V)
    with db.Graph(n, U, V) as g:
        db.fit_graph(g, iterations, 0.0)
        it, delta = db.fit_graph(g, 100, 1e-6)
        assert it + iterations == full["iterations"] and delta == full["delta"]
        np.testing.assert_array_equal(g.edge_dress.view(np.int64), full["edge_dress"].view(np.int64))


@pytest.mark.parametrize("bad", [0.0, -0.001, 1e-300, np.inf])
def test_a_weight_out_of_range_goes_the_other_way(bad, oracle_port):
    n, U, V = graphs.erdos_renyi(600, 3000, seed=11)
    W = np.random.default_rng(1).uniform(0.5, 2.0, 3000)
    W[1234] = bad
    _fit(oracle_port, n, U, V, W, one_launch=False)


def rows_that_depend_on_the_order(first, count, seed):
    """Weights of `count` rows whose sums after the term `first` are not the
    sorted Neumaier sums when the rounding errors are added up in the order
    given: `first` lies so far below the weights that the errors' sum loses it."""
    w = np.random.default_rng(seed).uniform(32, 64, (40_000, 16))
    x = np.concatenate([np.full((len(w), 1), first), w], axis=1)

    def total(x):
        s, c = x[:, 0].copy(), np.zeros(len(x))
        for j in range(1, x.shape[1]):
            t = s + x[:, j]
            b = t - s
            c = c + ((s - (t - b)) + (x[:, j] - b))
            s = t
        return np.sqrt(s + c)

    rows = w[total(x) != total(np.sort(x, axis=1))]
    assert len(rows) >= count
    return rows[:count]


@pytest.mark.parametrize("one_launch", [0, -1])
def test_vertex_weights_far_below_the_products(one_launch, oracle_port):
    """Self terms below the smallest product: errors are no multiples of its
    last place, and only a certificate shows that a sum is the sorted one."""
    first = 1.9 * 2.0 ** -97
    w = rows_that_depend_on_the_order(first, 80, 3)
    hub = np.arange(80)[:, None] * 17
    U = np.broadcast_to(hub, (80, 16)).astype(np.int32).ravel()
    V = (hub + np.arange(1, 17)).astype(np.int32).ravel()
    db.configure(one_launch_max_edges=one_launch)
    try:
        for iterations in (1, 100):
            _fit(oracle_port, 80 * 17, U, V, w.ravel(), np.full(80 * 17, first / 4), one_launch=None,
                 max_iterations=iterations)
    finally:
        db.configure()


def _certified(oracle_port, launches, *case, **kw):
    """_fit's comparison for fits that take `launches`: the pairs and certified
    sweeps, after an attempt within the range where that only shows on the way."""
    ref = oracle_port.fit(*case, **kw)
    variant = kw.pop("variant", db.UNDIRECTED)
    with db.Graph(*case, variant) as g:
        db.counters(reset=True)
        it, delta = db.fit_graph(g, **kw)
        assert launches is None or db.counters()["launches"] == launches
        assert (it, delta) == (ref["iterations"], ref["delta"])
        np.testing.assert_array_equal(g.edge_dress.view(np.int64), ref["edge_dress"].view(np.int64))
        np.testing.assert_array_equal(g.vertex_dress.view(np.int64), ref["vertex_dress"].view(np.int64))


@pytest.mark.parametrize("n,m", [(500, 1025), (700, 2049), (2000, 10000), (120, 4000), (9000, 16385), (400, 24001),
                                 (8000, 22000), (16000, 24575)])
@pytest.mark.parametrize("weights", ["one zero", "zeros", "signed", "tiny", "halves of zero vertices"])
def test_certified_sizes(n, m, weights, oracle_port):
    """The shapes of test_sizes off the range, in two launches."""
    n, U, V = graphs.erdos_renyi(n, m, seed=m)
    rng = np.random.default_rng(m)
    W = rng.uniform(0.5, 2.0, m)
    NW = None
    if weights == "one zero":
        W[m // 2] = 0.0
    elif weights == "zeros":
        W = rng.integers(0, 4, m).astype(float)
    elif weights == "signed":
        W = np.where(rng.random(m) < 0.05, -0.01, W)
    elif weights == "tiny":
        W[::3] = 1e-305
    else:
        W, NW = np.full(m, 0.5), rng.integers(0, 2, n).astype(float)
    _certified(oracle_port, 2, n, U, V, W, NW)


@pytest.mark.parametrize("variant", [db.UNDIRECTED, db.DIRECTED, db.FORWARD, db.BACKWARD])
@pytest.mark.parametrize("iterations", [1, 2, 3, 100])
def test_certified_variants_and_sweep_limits(variant, iterations, oracle_port):
    n, U, V = graphs.erdos_renyi(900, 5003, seed=7)
    rng = np.random.default_rng(variant)
    W = np.where(rng.random(5003) < 0.1, 0.0, rng.uniform(0.5, 2.0, 5003))
    _certified(oracle_port, 2, n, U, V, W, rng.uniform(0.3, 5.0, n), variant=variant, max_iterations=iterations)
    _certified(oracle_port, 2, n, U, V, W, None, variant=variant, max_iterations=iterations, epsilon=0.0)


@pytest.mark.parametrize("spread", [6.0, 7.0, 8.0])
def test_out_of_range_on_the_way(spread, oracle_port):
    """FORWARD rows with weights over many binades grow past the range."""
    n, U, V = graphs.erdos_renyi(900, 5003, seed=7)
    rng = np.random.default_rng(int(spread * 10))
    W = np.exp(rng.uniform(-spread, spread, 5003))
    NW = rng.uniform(0.3, 5.0, n)
    for kw in ({}, dict(epsilon=0.0), dict(max_iterations=60), dict(max_iterations=61)):
        _certified(oracle_port, 3, n, U, V, W, NW, variant=db.FORWARD, **kw)
    # up to the last sweep in range and past it, one launch and three
    for iterations in range(1, 40):
        _certified(oracle_port, None, n, U, V, W, NW, variant=db.FORWARD, max_iterations=iterations)


def test_values_out_of_range_to_go_on_from(oracle_port):
    """First values that put a product outside, which the host does not look for."""
    n, U, V = graphs.erdos_renyi(900, 5003, seed=7)
    d = np.ones(5003)
    d[17] = 1e-200
    ref = oracle_port.build(n, U, V)
    ctypes.memmove(ref.contents.edge_dress, d.ctypes.data, d.nbytes)
    it, delta = ctypes.c_int(), ctypes.c_double()
    oracle_port.fit_fn(ref, 100, 1e-6, ctypes.byref(it), ctypes.byref(delta))
    with db.Graph(n, U, V) as g:
        ctypes.memmove(g.ptr.contents.edge_dress, d.ctypes.data, d.nbytes)
        db.counters(reset=True)
        assert db.fit_graph(g) == (it.value, delta.value)
        assert db.counters()["launches"] == 3
        want = np.ctypeslib.as_array(ref.contents.edge_dress, shape=(5003,))
        np.testing.assert_array_equal(g.edge_dress.view(np.int64), want.view(np.int64))


@pytest.mark.parametrize("n,N,m", [(3000, 65_536, 2000), (400, 100_000, 900), (4000, 262_144, 4096), (60, 65_536, 1)])
@pytest.mark.parametrize("variant", [db.UNDIRECTED, db.FORWARD])
def test_few_edges_among_many_vertices(n, N, m, variant, oracle_port):
    """More vertices than 16-bit ids, most of them isolated (FORWARD: or without
    a row of their own): one launch, the isolated ones' norms among the results."""
    _, U, V = graphs.erdos_renyi(n, m, seed=m)
    rng = np.random.default_rng(m)
    at = rng.permutation(N)[:n].astype(np.int32)
    NW = rng.choice([0.5, 0.5, 0.0, 3.7], N)
    NW[at] = rng.uniform(0.5, 3.0, n)
    _fit(oracle_port, N, at[U], at[V], rng.uniform(0.5, 2.0, m), NW, variant)
    _fit(oracle_port, N, at[U], at[V], None, None, variant, max_iterations=2)


@pytest.mark.parametrize("n,N,m", [(3000, 262_145, 2000), (3000, 65_536, 4097)])
def test_many_vertices_beyond_the_one_launch(n, N, m, oracle_port):
    _, U, V = graphs.erdos_renyi(n, m, seed=2)
    _fit(oracle_port, N, U, V, one_launch=False)
