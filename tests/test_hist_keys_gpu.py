"""Histogram keys on the GPU: a run is one bit pattern.

The reference's map (libdress/src/dress_histogram.c:10-19, 40-60) hashes the
bit pattern of a value and merges by ==, so equal bit patterns always merge,
+0 and -0 (==-equal, different bits) land in different slots, and a NaN never
equals an entry.  The device histogram keeps +0 and -0 as two entries (-0
first) and every NaN apart; values are ascending, NaNs at the ends by bits.
"""
import ctypes

import numpy as np
import pytest

import dress_b200 as db
from dress_b200 import graphs

pytestmark = pytest.mark.gpu


def expected(values):
    k = values.view(np.uint64)
    order_key = np.where(k >> np.uint64(63) == 1, ~k, k | np.uint64(1 << 63))
    v = values[np.argsort(order_key, kind="stable")]
    out = []
    for x in v:
        b = int(np.float64(x).view(np.int64))
        if out and out[-2] == b and not np.isnan(x):
            out[-1] += 1
        else:
            out += [b, 1]
    return np.array(out, np.int64)


def test_signed_zeros_and_nans():
    import torch
    rng = np.random.default_rng(4)
    base = np.array([0.0, -0.0, 1.5, -2.0, np.inf, -np.inf, np.nan, 0.0, -0.0, 1.5, np.nan], np.float64)
    values = rng.permutation(np.concatenate([base, rng.choice(base[:6], 5000)]))
    dev = torch.device("cuda", 0)
    vals = torch.from_numpy(values).to(dev)
    pairs = torch.full((2 * values.size,), -1, dtype=torch.int64, device=dev)
    runs = torch.full((1,), -1, dtype=torch.int64, device=dev)
    stream = torch.cuda.current_stream(dev)
    rc = db.lib().dressx_histogram_noalloc(ctypes.c_void_p(vals.data_ptr()), values.size,
                                           ctypes.c_void_p(pairs.data_ptr()), ctypes.c_void_p(runs.data_ptr()),
                                           ctypes.c_void_p(stream.cuda_stream))
    assert rc == 0
    stream.synchronize()
    r = int(runs.item())
    got = pairs[: 2 * r].cpu().numpy()
    np.testing.assert_array_equal(got, expected(values))
    zeros = got.reshape(-1, 2)
    assert np.float64(-0.0).view(np.int64) in zeros[:, 0] and np.float64(0.0).view(np.int64) in zeros[:, 0]


def _runs(values):
    """expected(), vectorised (no NaN)."""
    k = values.view(np.uint64)
    key = np.where(k >> np.uint64(63) == 1, ~k, k | np.uint64(1 << 63))
    u, n = np.unique(key, return_counts=True)
    bits = np.where(u >> np.uint64(63) == 1, u & np.uint64((1 << 63) - 1), ~u)
    return np.stack([bits.view(np.int64), n], axis=1).ravel()


def _device_runs(values):
    import torch
    vals = torch.from_numpy(values).cuda()
    pairs = torch.full((2 * values.size + 3,), -7, dtype=torch.int64, device="cuda")
    runs = torch.zeros(1, dtype=torch.int64, device="cuda")
    out = pairs[1:]                                   # an int64 boundary is enough
    rc = db.lib().dressx_histogram_noalloc(ctypes.c_void_p(vals.data_ptr()), values.size,
                                           ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(runs.data_ptr()),
                                           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    r = int(runs.item())
    assert bool((vals.cpu() == torch.from_numpy(values)).all() or np.isnan(values).any())
    assert int(pairs[0]) == -7 and bool((out[2 * r:] == -7).all())      # nothing past the runs is written
    return out[: 2 * r].cpu().numpy()


def _values(kind, n, rng):
    if kind == "distinct":
        return rng.random(n)
    if kind == "few":
        return rng.random(7)[rng.integers(0, 7, n)]
    if kind == "constant":
        return np.full(n, 0.625)
    if kind == "one low bit":                         # keys that differ in the last bits of the mantissa only
        return (np.float64(1.25).view(np.int64) + rng.integers(0, 3, n)).view(np.float64)
    if kind == "signs":
        return rng.standard_normal(n) * np.exp(rng.uniform(-300, 300, n))
    v = rng.random(n)                                 # "heavy": one value fills most of the segment
    v[rng.random(n) < 0.9] = 0.3
    return v


@pytest.mark.parametrize("kind", ["distinct", "few", "constant", "one low bit", "signs", "heavy"])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 511, 512, 513, 8191, 8192, 8193, 12_289, 100_003, 1 << 20])
def test_sizes_of_a_segment(n, kind):
    """Around the block sizes of the bucket sort and of the split."""
    values = _values(kind, n, np.random.default_rng(n))
    np.testing.assert_array_equal(_device_runs(values), _runs(values))


def test_a_sample_that_misses_every_value_but_one():
    """Splitters come from jittered places; with one value at all of them the
    rest falls into one bucket, far beyond what a block sorts in shared memory."""
    n, ns = 1 << 20, 8 * 512
    p = np.arange(ns, dtype=np.uint64)
    h = (p * np.uint64(2654435761)) & np.uint64(0xffffffff)
    h ^= h >> np.uint64(15)
    h = (h * np.uint64(2246822519)) & np.uint64(0xffffffff)
    h ^= h >> np.uint64(13)
    at = (p * np.uint64(n // ns) + h % np.uint64(n // ns)).astype(np.int64)
    rng = np.random.default_rng(1)
    for below, above in ((True, False), (False, True)):
        values = np.where(rng.random(n) < 0.5, rng.random(n), rng.integers(0, 50, n) / 64.0)
        values = values if below else values + 2.0
        values[at] = 1.5
        np.testing.assert_array_equal(_device_runs(values), _runs(values))


def test_nans_in_a_long_segment():
    rng = np.random.default_rng(2)
    values = rng.random(40_000)
    values[rng.random(values.size) < 0.6] = np.nan
    got = _device_runs(values).reshape(-1, 2)
    nans = np.isnan(got[:, 0].copy().view(np.float64))
    assert nans.sum() == np.isnan(values).sum() and bool((got[nans, 1] == 1).all())
    np.testing.assert_array_equal(got[~nans].ravel(), _runs(values[~np.isnan(values)]))


def test_segments_of_every_size_at_once(oracle_port):
    """Segments of one bucket and split ones in one call."""
    gs = []
    for i, (n, d) in enumerate([(16, 3), (60, 8), (100, 6), (130, 12), (200, 10), (18, 4)]):
        gs.append(graphs.random_regular(n, d, seed=i))
    objs = [db.Graph(*g) for g in gs]
    for g, flat in zip(gs, db.delta_fit_many(objs, k=1)):
        np.testing.assert_array_equal(flat, oracle_port.delta_fit(*g, k=1)["hist"])
    for o in objs:
        o.close()




def _shares(g, n, k, parts, **kw):
    """The histogram of a request and the merged ones of its strided shares."""
    from dress_b200 import shard
    whole, _, _, fits, _ = db.hist_requests([g], db.DELTA, k, **kw)[0]
    flats = [db.hist_requests([g], db.DELTA, k, offset=i, stride=parts, **kw)[0][0] for i in range(parts)]
    return whole, shard.merge_hists(flats), fits


@pytest.mark.parametrize("n,parts", [(140, 4), (200, 24), (300, 80)])
def test_long_segments_of_distinct_values(n, parts):
    """6.6, 19.5 and 66 million mostly distinct values: 4,096 buckets of which
    few, a part and nearly all are more than a block holds.  The shares have at
    most two million values, with buckets that a block holds."""
    g = db.Graph(*graphs.random_regular(n, 10, seed=9))
    whole, merged, _ = _shares(g, n, 2, parts, max_iterations=4)
    assert whole.size > 10_000_000
    np.testing.assert_array_equal(whole, merged)
    g.close()


@pytest.mark.slow
def test_a_segment_of_more_values_than_32_bits_count():
    """Delta^2 of a circulant graph of 1,000 vertices and 9,000 edges: 4.5*10^9
    values, taken in pieces.  Each of its three shares is one piece."""
    import torch
    if torch.cuda.mem_get_info()[0] < 120 << 30:
        pytest.skip("needs 85 GB of device memory")
    n = 1000
    U = np.tile(np.arange(n, dtype=np.int32), 9)
    V = np.concatenate([(np.arange(n) + c) % n for c in range(1, 10)]).astype(np.int32)
    g = db.Graph(n, U, V)
    whole, merged, fits = _shares(g, n, 2, 3, max_iterations=2)
    assert fits == n * (n - 1) // 2
    assert int(whole[1::2].sum()) == fits * 9 * n - sum(2 * 18 - (1 if min(d, n - d) < 10 else 0)
                                                          for d in range(1, n)) * n // 2
    np.testing.assert_array_equal(whole, merged)
    g.close()
