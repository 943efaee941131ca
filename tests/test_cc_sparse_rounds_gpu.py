"""Connected components on few edges per vertex: rounds on all edges and on the list of the open ones."""
import numpy as np
import pytest

import pyoracle as O

pytestmark = pytest.mark.gpu

FEW = 1 << 18  # edges from which on one more round is allowed


def _random(n, m, seed=1):
    rng = np.random.default_rng(seed + n + m)
    return n, rng.integers(0, n, m), rng.integers(0, n, m)


def _relabelled(n, u, v):
    rng = np.random.default_rng(2)
    q, p = rng.permutation(n), rng.permutation(len(u))
    return n, q[u][p], q[v][p]


def _tree(n):
    i = np.arange(1, n)
    return n, (i * np.random.default_rng(3).random(n - 1)).astype(np.int64), i


def _star(n, hub):
    return n, np.full(n - 1, hub), np.delete(np.arange(n), hub)


def _path(n):
    return n, np.arange(n - 1), np.arange(1, n)


CASES = {
    "smallest": _random(16321, 8193),
    "degree just below 1": _random(20002, 10000),
    "degree 1": _random(20000, 10000),
    "degree below 1.2": _random(50000, 29999),
    "degree 1.2": _random(50000, 30000),
    "below the line of degrees": _random(50000, 59999),
    "above it": _random(50000, 60001),
    "threshold of the giant": _random(200003, 110000),
    "one round fewer": _random(250001, FEW - 1),
    "one round more": _random(250001, FEW),
    "wide CTAs": _random(1500001, 1600013),
    "one edge in the last tile": _random(100000, 256 * 400 + 1),
    "path": _path(300007),
    "path relabelled": _relabelled(*_path(300007)),
    "star at 0": _star(100001, 0),
    "star at the last": _star(300001, 300000),
    "star relabelled": _relabelled(*_star(300001, 0)),
    "tree relabelled": _relabelled(*_tree(400009)),
    "matching": (200000, np.arange(0, 200000, 2), np.arange(1, 200000, 2)),
    "loops and twice the same": (30000, np.tile(np.arange(15000), 2), np.tile(np.arange(15000) // 3, 2)),
}


@pytest.mark.parametrize("case", CASES)
def test_labels(ctx, case):
    n, u, v = CASES[case]
    u, v = u.astype(np.uint32), v.astype(np.uint32)
    want_count, want = O.cc_labels(n, u, v)
    g = ctx.graph(n, u, v)
    for ranks in (1, 1, 1, 7):  # direct, captured, replayed, direct
        count, lab, _ = g.connected_components(seed=1, virtual_ranks=ranks)
        assert count == want_count and np.array_equal(lab, want)
    lab = np.zeros(n, np.uint32)
    assert ctx.cc_edges(n, u, v, labels=lab).num_components == want_count
    assert np.array_equal(lab, want)


@pytest.mark.parametrize("n,m", [(100000, 100000), (1000000, 1000000)])
def test_bad_endpoints(ctx, libcac, n, m):
    _, u, v = _random(n, m)
    u, v = u.astype(np.uint32), v.astype(np.uint32)
    for at in (0, m // 3, m - 1):
        bad = v.copy()
        bad[at] = n
        with pytest.raises(libcac.CacError) as e:
            ctx.cc_edges(n, u, bad)
        assert e.value.status == -1
    want_count, _ = O.cc_labels(n, u, v)
    assert ctx.cc_edges(n, u, v).num_components == want_count


def test_time_near_the_threshold_of_a_giant_component(ctx):
    # degree 2 has two thirds of the edges of degree 3 and at most one more round and compression (about 20 us of
    # 120): about as long. Left to union walks, its open edges between few large trees take three times as long.
    n, times = 1000000, []
    for degree in (2, 3):
        t = []
        for seed in range(3):
            _, u, v = _random(n, n * degree // 2, seed)
            g = ctx.graph(n, u.astype(np.uint32), v.astype(np.uint32))
            t += [g.connected_components(seed=9, labels=False)[2].device_ms for _ in range(5)][2:]
        times.append(float(np.median(t)))
    assert times[0] < 2 * times[1], times


def test_more_vertices_than_the_rounds_on_lists_take(ctx):
    # 2^24 and one more; the labels by the device generator's graph and the oracle
    for n in (1 << 24, (1 << 24) + 1):
        g = ctx.generate("erdos_renyi_m", seed=5, n=n, avg_degree=1.3, wmax=1)
        u, v, _ = g.edges()
        want_count, want = O.cc_labels(n, u, v)
        count, lab, _ = g.connected_components(seed=1, virtual_ranks=2)
        assert count == want_count and np.array_equal(lab, want)
