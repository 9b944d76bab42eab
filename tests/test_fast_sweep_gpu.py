"""The multi-kernel fit's fast sweeps, bit for bit against the oracle: every
class of rows and edges (a thread, 8, 16, 32 lanes, a block), and fits that
leave the fast range at the start, in the middle, or never."""
import numpy as np
import pytest

import dress_b200 as db
from dress_b200 import graphs

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def multi_kernel():
    db.configure(one_launch_max_edges=-1)
    yield
    db.configure()


def _fit(oracle_port, n, U, V, W=None, NW=None, variant=db.UNDIRECTED, **kw):
    ref = oracle_port.fit(n, U, V, W, NW, variant=variant, **kw)
    with db.Graph(n, U, V, W, NW, variant) as g:
        it, delta = db.fit_graph(g, kw.get("max_iterations", 100), kw.get("epsilon", 1e-6))
        assert (it, delta) == (ref["iterations"], ref["delta"])
        np.testing.assert_array_equal(g.edge_dress.view(np.int64), ref["edge_dress"].view(np.int64))
        np.testing.assert_array_equal(g.vertex_dress.view(np.int64), ref["vertex_dress"].view(np.int64))


def _dense_core(rng):
    """A core of 1,100 vertices joined at random (rows of 500 to 700, as many
    common neighbours as pairs of a thread to a block take), two hubs over all
    of 6,000 vertices, and sparse rest."""
    core = np.argwhere(np.triu(rng.random((700, 700)) < 0.4, 1))
    thin = np.argwhere(np.triu(rng.random((400, 400)) < 0.08, 1)) + 700
    hubs = [(6000 + h, x) for h in range(2) for x in range(6000)] + [(6000, 6001)]
    rest = rng.integers(1100, 6000, (8000, 2))
    e = np.concatenate([core, thin, np.array(hubs), rest])
    e = np.sort(e[e[:, 0] != e[:, 1]], axis=1)
    e = np.unique(e, axis=0)
    e = e[rng.permutation(len(e))].astype(np.int32)
    return 6002, e[:, 0].copy(), e[:, 1].copy()


@pytest.mark.parametrize("weights", ["none", "uniform", "third"])
def test_every_class(weights, oracle_port):
    rng = np.random.default_rng(1)
    n, U, V = _dense_core(rng)
    m = len(U)
    W = {"none": None, "uniform": rng.uniform(0.5, 2.0, m), "third": np.full(m, 0.3)}[weights]
    NW = rng.uniform(0.5, 2.0, n) if weights == "uniform" else None
    _fit(oracle_port, n, U, V, W, NW)


@pytest.mark.parametrize("m", [1, 2, 255, 256, 257, 5000, 30001])
def test_sizes(m, oracle_port):
    n, U, V = graphs.erdos_renyi(max(3, m // 3), m, seed=m)
    _fit(oracle_port, n, U, V, np.random.default_rng(m).uniform(0.5, 2.0, m))


@pytest.mark.parametrize("iterations", [1, 2, 5, 9, 33])
def test_sweep_limits(iterations, oracle_port):
    n, U, V = graphs.chung_lu(900, 6000, 2.3, 400, seed=3)
    _fit(oracle_port, n, U, V, max_iterations=iterations, epsilon=0.0)


@pytest.mark.parametrize("bad", [0.0, -0.001, 1e-300])
def test_out_of_range_from_the_start(bad, oracle_port):
    n, U, V = graphs.chung_lu(900, 6000, 2.3, 400, seed=3)
    W = np.random.default_rng(2).uniform(0.5, 2.0, 6000)
    W[::7] = bad
    _fit(oracle_port, n, U, V, W)


@pytest.mark.parametrize("variant", [db.FORWARD, db.BACKWARD])
@pytest.mark.parametrize("spread", [4.0, 5.0, 6.0, 7.0, 8.0])
@pytest.mark.parametrize("iterations", [9, 100])
def test_out_of_range_on_the_way(variant, spread, iterations, oracle_port):
    """Directed rows with weights over many binades grow for dozens of sweeps;
    the certified sweeps take over at an even or an odd one."""
    n, U, V = graphs.erdos_renyi(900, 5003, seed=7)
    rng = np.random.default_rng(int(spread * 10))
    W = np.exp(rng.uniform(-spread, spread, 5003))
    NW = rng.uniform(0.3, 5.0, n)
    _fit(oracle_port, n, U, V, W, NW, variant, max_iterations=iterations)


@pytest.mark.parametrize("loops", [0, 3])
def test_large_renumbering(loops, oracle_port):
    """2^20 edges and more are renumbered by owner from the oriented rows, with
    a self loop (which is in none) by sorted keys; rows of 1 to 1,500 slots."""
    n, U, V = graphs.chung_lu(150_001, (1 << 20) + 5, 2.3, 1500, seed=4)
    V[:loops] = U[:loops]
    _fit(oracle_port, n, U, V, np.random.default_rng(5).uniform(0.5, 2.0, len(U)), max_iterations=4)


@pytest.mark.parametrize("low", [2, 31, 32, 33, 511, 512, 513, 700])
def test_owner_rows(low, oracle_port):
    """A vertex whose oriented row has `low` members (hashed up to 512, then
    searched), all of them of higher degree and some joined to each other."""
    rng = np.random.default_rng(low)
    core = np.arange(1, low + 1)
    far = np.arange(low + 1, 2 * low + 41)
    e = [np.stack([np.zeros(low, int), core], 1)]
    e += [np.stack([np.full(low + 1, c), rng.choice(far, low + 1, replace=False)], 1) for c in core]
    for _ in range(2):
        e.append(np.stack([core, rng.permutation(core)], 1))
    e = np.concatenate(e)
    e = np.unique(np.sort(e[e[:, 0] != e[:, 1]], axis=1), axis=0)
    e = e[rng.permutation(len(e))].astype(np.int32)
    _fit(oracle_port, int(e.max()) + 1, e[:, 0].copy(), e[:, 1].copy(), max_iterations=5)


@pytest.mark.parametrize("zero", [0.0, -0.0])
def test_zero_weights_keep_the_fast_sweeps(zero, oracle_port):
    """Zero products change no sum: ten sweeps take the launches that they take
    without zeros.  A first product outside leaves no sweep to the fast kernels."""
    n, U, V = graphs.chung_lu(900, 6000, 2.3, 400, seed=3)
    W = np.random.default_rng(2).uniform(0.5, 2.0, 6000)
    launches = []
    for w in (1.0, zero, -0.001):
        W[::7] = w
        with db.Graph(n, U, V, W) as g:
            db.counters(reset=True)
            db.fit_graph(g, 10, 0.0)
            launches.append(db.counters()["launches"])
        _fit(oracle_port, n, U, V, W)
        _fit(oracle_port, n, U, V, W, np.random.default_rng(3).uniform(0.5, 2.0, n), db.FORWARD)
    assert launches[0] == launches[1] < launches[2]


@pytest.mark.parametrize("joins", [2, 7])
def test_owner_rows_beyond_the_ranked(joins, oracle_port):
    """More than 2^20 edges and an oriented row of more than 1,024: that row keeps
    its order in the renumbering by owner.  With seven permutations of the core
    joined the triangles overflow their list, and a second pass makes the pairs."""
    low = 1100
    rng = np.random.default_rng(joins)
    core = np.arange(1, low + 1)
    far = np.arange(low + 1, 2 * low + 41)
    e = [np.stack([np.zeros(low, int), core], 1)]
    e += [np.stack([np.full(low + 1, c), rng.choice(far, low + 1, replace=False)], 1) for c in core]
    e += [np.stack([core, rng.permutation(core)], 1) for _ in range(joins)]
    e = np.concatenate(e)
    e = np.unique(np.sort(e[e[:, 0] != e[:, 1]], axis=1), axis=0)
    e = e[rng.permutation(len(e))].astype(np.int32)
    assert len(e) > 1 << 20
    _fit(oracle_port, int(e.max()) + 1, e[:, 0].copy(), e[:, 1].copy(), rng.uniform(0.5, 2.0, len(e)), max_iterations=1)


@pytest.mark.parametrize("n,variant", [(520, db.UNDIRECTED), (330, db.UNDIRECTED), (520, db.FORWARD)])
def test_many_long_lists_of_pairs(n, variant, oracle_port):
    """A complete graph: 134,940 edges of 518 pairs are a warp each, 54,285 of
    328 lane groups as ever."""
    U, V = (x.astype(np.int32) for x in np.triu_indices(n, 1))
    W = np.random.default_rng(n).uniform(0.5, 2.0, len(U))
    _fit(oracle_port, n, U, V, W, variant=variant, max_iterations=2)
