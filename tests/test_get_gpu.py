"""Virtual-edge queries where their kernels change shape, bit for bit against
the oracle: rows around a warp's width, a hub, parallel edges, queries of
existing edges and of a vertex with itself, and the pairs whose sums take the
sorted path."""
import numpy as np
import pytest

import dress_b200 as db
from dress_b200 import graphs

pytestmark = pytest.mark.gpu


def _bipartite_rows(sizes, rng):
    """Vertices 0 and 1 share `sizes[i]` neighbours with vertex 2 + i."""
    U, V, n = [], [], 2 + len(sizes)
    for i, s in enumerate(sizes):
        for x in range(n, n + s):
            U += [0, 2 + i]
            V += [x, x]
        n += s
    p = rng.permutation(len(U))
    return n, np.array(U, np.int32)[p], np.array(V, np.int32)[p]


def _check(oracle_port, n, U, V, W, q, variant=db.UNDIRECTED):
    ref = oracle_port.get_many(n, U, V, W, q, 100, 1e-6, 0.8, variant=variant)
    with db.Graph(n, U, V, W, variant=variant) as g:
        db.fit_graph(g, 100, 1e-6)
        got = db.get(g, [a for a, _ in q], [b for _, b in q], 100, 1e-6, 0.8)
    np.testing.assert_array_equal(got.view(np.int64), ref.view(np.int64))


@pytest.fixture(params=[0, 1], ids=["certified", "sorted"])
def exact(request):
    db.configure(exact_sums=request.param)
    yield request.param
    db.configure()


@pytest.mark.parametrize("variant", [db.UNDIRECTED, db.DIRECTED, db.FORWARD, db.BACKWARD])
def test_rows_around_a_warp(exact, variant, oracle_port):
    rng = np.random.default_rng(3)
    sizes = [1, 2, 31, 32, 33, 63, 64, 65, 200]
    n, U, V = _bipartite_rows(sizes, rng)
    W = rng.uniform(0.5, 2.0, len(U))
    q = [(0, 2 + i) for i in range(len(sizes))] + [(2 + i, 0) for i in range(len(sizes))]
    q += [(2, 3), (0, 0), (1, 1), (0, 1), (2, n - 1), (int(U[5]), int(V[5])), (int(V[7]), int(U[7]))]
    _check(oracle_port, n, U, V, W, q, variant)


@pytest.mark.parametrize("weights", ["none", "uniform", "signed"])
def test_multigraph(exact, weights, oracle_port):
    """Rows with runs of parallel edges: the i-th of a run meets the i-th."""
    rng = np.random.default_rng(4)
    m = 900
    U = rng.integers(0, 25, m).astype(np.int32)
    V = rng.integers(0, 25, m).astype(np.int32)
    W = {"none": None, "uniform": rng.uniform(0.5, 2.0, m), "signed": rng.choice([-0.01, 0.0, 1.0, 2.0], m)}[weights]
    q = [(int(a), int(b)) for a in range(25) for b in range(25)]
    _check(oracle_port, 25, U, V, W, q)


def test_power_law_pairs(exact, oracle_port):
    n, U, V = graphs.chung_lu(600, 4200, 2.3, 300, seed=2)
    rng = np.random.default_rng(5)
    q = list(zip(rng.integers(0, n, 300).tolist(), rng.integers(0, n, 300).tolist()))
    _check(oracle_port, n, U, V, None, q)


@pytest.mark.parametrize("run,other", [(31, 33), (64, 40), (1000, 999), (1500, 1600)])
def test_long_runs_of_parallel_edges(run, other, oracle_port):
    """Runs within, across and far beyond a warp's strip, of unequal length in
    the two rows; the place in a run is found by search, not step by step."""
    rng = np.random.default_rng(run)
    U = np.concatenate([np.zeros(3 * run), np.ones(3 * other), [0, 1]]).astype(np.int32)
    V = np.concatenate([np.repeat([2, 3, 5], run), np.repeat([2, 4, 5], other), [6, 6]]).astype(np.int32)
    p = rng.permutation(len(U))
    _check(oracle_port, 7, U[p], V[p], rng.uniform(0.5, 2.0, len(U)), [(0, 1), (1, 0), (2, 6), (0, 6)])
