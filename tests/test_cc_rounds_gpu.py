"""Connected components in one CTA (small graphs) and by rounds of root links: labels against the oracle's."""
import numpy as np
import pytest

import graphgen
import pyoracle as O

pytestmark = pytest.mark.gpu

SMALL_N, SMALL_M = (64 * 1024 - 256) // 4, 1 << 16  # the one-CTA form's limits


def _check(ctx, n, u, v, **kw):
    want_count, want = O.cc_labels(n, u, v)
    g = ctx.graph(n, u, v)
    for seed in (0, 3):
        count, lab, _ = g.connected_components(seed=seed, **kw)
        assert count == want_count and np.array_equal(lab, want)
    count, _, _ = g.connected_components(seed=1, labels=False, **kw)
    assert count == want_count
    return g, want_count, want


@pytest.mark.parametrize("n,m", [
    (1, 0), (2, 1), (31, 40), (1023, 700), (1024, 4096), (1025, 1200), (SMALL_N, 12000), (SMALL_N, SMALL_M),
    (SMALL_N, SMALL_M + 1), (SMALL_N + 1, SMALL_M), (SMALL_N + 1, 8191), (SMALL_N + 1, 8192),
])
def test_limits_of_the_one_cta_form(ctx, n, m):
    rng = np.random.default_rng(n + m)
    u, v = (rng.integers(0, n, m).astype(np.uint32) for _ in range(2))
    _check(ctx, n, u, v, virtual_ranks=2)


def test_one_cta_form_outputs_and_bad_endpoints(ctx, libcac):
    torch = pytest.importorskip("torch")
    import cac
    n, u, v, _ = graphgen.rmat(12, 4, 5)
    want_count, want = O.cc_labels(n, u, v)
    out = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert ctx.graph(n, u, v).connected_components(out=out)[0] == want_count
    assert np.array_equal(out.cpu().numpy().view(np.uint32), want)
    lab = np.zeros(n, np.uint32)
    assert ctx.cc_edges(n, u, v, labels=lab).num_components == want_count and np.array_equal(lab, want)
    assert ctx.cc_edges(n, u, v).num_components == want_count
    for at in (0, len(u) // 2, len(u) - 1):
        bad = v.copy()
        bad[at] = n
        with pytest.raises(cac.CacError):
            ctx.cc_edges(n, u, bad, labels=lab)


def _path(n):
    return n, np.arange(n - 1), np.arange(1, n)


def _grid(w, h):
    i = np.arange(w * h).reshape(h, w)
    return w * h, np.concatenate([i[:, :-1].ravel(), i[:-1].ravel()]), np.concatenate([i[:, 1:].ravel(), i[1:].ravel()])


def _ring(n, k):
    i = np.arange(n)
    return n, np.concatenate([i] * k), np.concatenate([(i + d) % n for d in range(1, k + 1)])


def _hubs(n):  # three hubs with the largest, a middle and the smallest id, every edge four times
    i = np.arange(n)
    u = np.concatenate([np.full(n, n - 1), np.full(n, n // 2), np.zeros(n, np.int64)])
    v = np.concatenate([i % 1000, i, n - 1 - i // 7])
    return n, np.tile(u, 4), np.tile(v, 4)


@pytest.mark.parametrize("shape", ["path", "path reversed", "grid", "ring", "hubs", "matching"])
@pytest.mark.parametrize("shuffled", [False, True])
def test_rounds_on_structured_graphs(ctx, shape, shuffled):
    # vertices numbered along a path make parent chains as long as it (compressions stop short of the
    # root); hubs and large trees gather thousands of links in one round
    n, u, v = {"path": lambda: _path(70001), "path reversed": lambda: _path(70001), "grid": lambda: _grid(301, 203),
               "ring": lambda: _ring(40003, 6), "hubs": lambda: _hubs(50002),
               "matching": lambda: (80003, np.arange(0, 80000, 2), np.arange(1, 80001, 2))}[shape]()
    if shape == "path reversed":
        u, v = n - 1 - u, n - 1 - v
    if shuffled:
        p = np.random.default_rng(1).permutation(len(u))
        u, v = u[p], v[p]
    _check(ctx, n, u.astype(np.uint32), v.astype(np.uint32), virtual_ranks=3)


@pytest.mark.parametrize("n,degree", [(20001, 0.9), (20002, 1.1), (60003, 2.0), (60000, 4.9), (100001, 7.3), (17000, 40.0)])
def test_rounds_over_densities(ctx, n, degree):
    # from single-pass (degree < 1) over rounds on all edges to rounds on drawn chunks
    _, u, v, _ = graphgen.erdos_renyi_m(n, degree, 11, wmax=1)
    _check(ctx, n, u, v, virtual_ranks=5)
    lab = np.zeros(n, np.uint32)
    want_count, want = O.cc_labels(n, u, v)
    assert ctx.cc_edges(n, u, v, virtual_ranks=5, labels=lab).num_components == want_count
    assert np.array_equal(lab, want)


def test_labels_with_more_tiles_than_a_ranking_cta_sums(ctx):
    n = 4096 * 1024 + 5  # one tile more than kOwnTiles
    rng = np.random.default_rng(2)
    u, v = (rng.integers(0, n, 3000000).astype(np.uint32) for _ in range(2))
    _check(ctx, n, u, v)
