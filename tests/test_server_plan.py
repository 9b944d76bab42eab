"""Host-side planning of served requests (no GPU, but for one test): path choice
and the device bytes a request reserves at admission."""
import ctypes

import numpy as np
import pytest

import dress_b200 as db
from dress_b200 import graphs

EINVAL = 1


def test_small_graphs_take_the_batch_path():
    n, U, V = graphs.random_regular(100, 6, seed=1)
    with db.Graph(n, U, V) as g:
        b_fit, p_fit = db.estimate(g, db.FIT)
        b_delta, p_delta = db.estimate(g, db.DELTA, 1)
        b_nabla, p_nabla = db.estimate(g, db.NABLA, 1)
    assert p_fit == p_delta == p_nabla == db.PATH_BATCH
    # a fit holds its graph and outputs; a Delta^1 request also its 100 x 300
    # subgraph values and their histogram scratch
    assert 0 < b_fit < b_delta
    assert b_delta >= 100 * 300 * 8 * 2
    assert b_nabla == b_delta


def test_hub_rows():
    # hub rows: the whole-graph fit runs on the single-graph engine (a warp or
    # a block per long row); the Delta^1 subgraphs are batched, their rows of
    # any length summed in the batch kernel
    n, U, V = graphs.chung_lu(2000, 6000, 2.3, 500, seed=2)
    with db.Graph(n, U, V) as g:
        assert max(np.diff(g.ptr.contents.adj_offset[: n + 1])) > 256
        assert db.estimate(g, db.FIT)[1] == db.PATH_LANE
        assert db.estimate(g, db.DELTA, 1)[1] == db.PATH_BATCH


def test_trivial_orders_take_a_lane():
    n, U, V = graphs.random_regular(40, 4, seed=3)
    with db.Graph(n, U, V) as g:
        assert db.estimate(g, db.DELTA, 0)[1] == db.PATH_LANE     # k = 0 fits in place
        assert db.estimate(g, db.DELTA, 40)[1] == db.PATH_LANE    # k >= N: empty histogram


def test_state_beyond_shared_memory_takes_a_lane():
    # 4-regular with 20000 edges: rows are short but one subgraph's state
    # (2 x 20000 edge values + norms) exceeds shared memory
    n, U, V = graphs.random_regular(10000, 4, seed=4)
    with db.Graph(n, U, V) as g:
        assert db.estimate(g, db.DELTA, 1)[1] == db.PATH_LANE


def test_larger_whole_graph_fits_take_a_lane():
    # 3000 edges: its Delta^1 subgraphs are batched, the whole-graph fit runs
    # on the single-graph engine, which spreads each sweep over the device
    n, U, V = graphs.random_regular(1000, 6, seed=4)
    with db.Graph(n, U, V) as g:
        assert db.estimate(g, db.FIT)[1] == db.PATH_LANE
        assert db.estimate(g, db.DELTA, 1)[1] == db.PATH_BATCH


def test_estimate_grows_with_the_graph():
    sizes = []
    for n in (50, 200, 800):
        nn, U, V = graphs.random_regular(n, 4, seed=5)
        with db.Graph(nn, U, V) as g:
            sizes.append(db.estimate(g, db.DELTA, 1)[0])
    assert sizes[0] < sizes[1] < sizes[2]


def test_malformed_requests_are_refused():
    n, U, V = graphs.random_regular(20, 4, seed=6)
    with db.Graph(n, U, V) as g:
        for kind, k in ((7, 0), (db.DELTA, -1)):
            try:
                db.estimate(g, kind, k)
            except db.DressError as e:
                assert e.code == EINVAL
            else:
                raise AssertionError("accepted a malformed request")
        g.ptr.contents.U[2] = 99         # endpoint out of range
        try:
            db.estimate(g, db.FIT)
        except db.DressError as e:
            assert e.code == EINVAL
        else:
            raise AssertionError("accepted an out-of-range endpoint")
        g.ptr.contents.U[2] = U[2]


def test_a_histogram_reserves_what_it_takes():
    # 8 bytes a value twice, 2 of bucket ids, at most 16 of runs, and little else
    n, U, V = graphs.random_regular(200, 10, seed=1)
    with db.Graph(n, U, V) as g:
        for k in (1, 2):
            values = n * (n - 1) // 2 * 1000 if k == 2 else n * 1000
            per_value = db.estimate(g, db.DELTA, k)[0] / values
            assert 34 <= per_value < 37


def own_rows(c, n, per_row):
    """Rows of a caller's own for the cycle of n vertices, each neighbour listed
    per_row / 2 times; returns what puts the graph's rows back."""
    u = np.arange(n, dtype=np.int32)
    nbr, eid = np.stack([np.roll(u, 1), np.roll(u, -1)], 1), np.stack([np.roll(u, 1), u], 1)
    order = np.argsort(nbr, axis=1)
    tgt, idx = (np.repeat(np.take_along_axis(a, order, 1), per_row // 2, axis=1).ravel() for a in (nbr, eid))
    rows = {"adj_offset": np.arange(0, n * per_row + 1, per_row, dtype=np.int32),
            "adj_target": tgt, "adj_edge_idx": idx}
    ip = ctypes.POINTER(ctypes.c_int)
    kept = {f: ctypes.cast(getattr(c, f), ctypes.c_void_p).value for f in rows}
    for f, a in rows.items():
        setattr(c, f, a.ctypes.data_as(ip))
    c.max_degree = per_row                               # what the oracle's buffer is sized by

    def back():
        for f, p in kept.items():
            setattr(c, f, ctypes.cast(p, ip))
        return rows

    return back


# the batch kernel's image names 65,535 groups of four slots
ROWS = [(200, db.PATH_BATCH), (216, db.PATH_LANE), (256, db.PATH_LANE)]


@pytest.mark.parametrize("per_row, path", ROWS)
def test_rows_of_more_slots_than_the_image_names(per_row, path):
    n = 1200
    U = np.arange(n, dtype=np.int32)
    with db.Graph(n, U, np.roll(U, -1)) as g:
        back = own_rows(g.ptr.contents, n, per_row)
        paths = [db.estimate(g, kind, k)[1] for kind, k in ((db.FIT, 0), (db.DELTA, 1))]
        back()
    assert paths == [path, path]


@pytest.mark.gpu
@pytest.mark.parametrize("per_row, path", ROWS)
def test_served_fit_of_own_rows(per_row, path, oracle_port):
    n = 1200
    U = np.arange(n, dtype=np.int32)
    V = np.roll(U, -1)
    W = np.random.default_rng(1).uniform(0.5, 2.0, n)
    ref = oracle_port.build(n, U, V, W, None, db.UNDIRECTED, 0)
    back = own_rows(ref.contents, n, per_row)
    it, delta = ctypes.c_int(), ctypes.c_double()
    oracle_port.fit_fn(ref, 100, 1e-6, ctypes.byref(it), ctypes.byref(delta))
    want = [np.ctypeslib.as_array(f, shape=(n,)).copy() for f in (ref.contents.edge_dress, ref.contents.vertex_dress)]
    back()
    oracle_port.free_graph(ref)
    with db.Server() as srv, db.Graph(n, U, V, W) as g:
        back = own_rows(g.ptr.contents, n, per_row)
        r = srv.submit(g).wait()
        back()
        assert r["status"] == 0 and r["path"] == path
        assert (r["iterations"], r["delta"]) == (it.value, delta.value)
        for a, b in zip((g.edge_dress, g.vertex_dress), want):
            np.testing.assert_array_equal(a.view(np.int64), b.view(np.int64))
