"""The leaf solver (one warp, four vertices per lane, lower triangle) at its edges, against the oracle's exact cut."""
import numpy as np
import pytest

import pyoracle as O

pytestmark = pytest.mark.gpu


def _clusters(n, parts, weight, seed):
    """Cliques of random weights joined in a ring by unit edges: orderings end with several clusters left, so
    vertices are merged and later orderings start from merged rows."""
    rng = np.random.default_rng(seed)
    home = rng.permutation(np.arange(n) % parts)  # members of a cluster in every group of 32 vertices
    w = np.triu(rng.integers(1, weight, (n, n), endpoint=True).astype(np.uint64) * (home[:, None] == home), 1)
    w += w.T
    first = [int(np.flatnonzero(home == c)[0]) for c in range(parts)]
    for c in range(parts):
        a, b = first[c], first[(c + 1) % parts]
        if a != b:
            w[a, b] += np.uint64(1)
            w[b, a] = w[a, b]
    return w


# the entry and vertex-word widths: 32/32 bits, 32/64 (total weight 2^24 and more), 64/64
@pytest.mark.parametrize("weight", [3, 1 << 20, 1 << 33])
@pytest.mark.parametrize("parts", [1, 2, 5, 16])
@pytest.mark.parametrize("n", [2, 3, 31, 32, 33, 64, 65, 96, 97, 127, 128])
def test_leaf_matches_exact_cut(ctx, n, parts, weight):
    mat = _clusters(n, min(parts, n), weight, 7 * n + parts)
    assert ctx.exact_cut_small(mat) == O.stoer_wagner_dense(mat)


def test_leaf_path_and_star(ctx):
    # a path is contracted along one chain of certified edges, 127 long
    n = 128
    path = np.zeros((n, n), np.uint64)
    i = np.arange(n - 1)
    path[i, i + 1] = path[i + 1, i] = 5 + i % 7
    star = np.zeros((n, n), np.uint64)
    star[0, 1:] = star[1:, 0] = 9
    for mat in (path, path[::-1, ::-1].copy(), star):
        assert ctx.exact_cut_small(mat) == O.stoer_wagner_dense(mat)


# leaves solved straight from their source: 1 to 51 joined vertices, above 179 none; both entry widths,
# groups of one to dozens of members, planned ahead (a graph's trials) and level by level (a matrix)
@pytest.mark.parametrize("wmax", [9, 1 << 20, 1 << 31])
@pytest.mark.parametrize("hub", [False, True])
@pytest.mark.parametrize("n", [129, 130, 159, 160, 161, 178, 179, 180, 181])
def test_trial_with_leaf_children(ctx, n, hub, wmax):
    rng = np.random.default_rng(n + hub)
    u, v = np.triu_indices(n, 1)
    w = rng.integers(1, wmax, len(u), endpoint=True).astype(np.uint64)
    if hub:  # most draws join a few vertices
        heavy = (v < 12) | (rng.random(len(u)) < 0.01)
        w = np.where(heavy, w, w // 9 + 1)
    keep = rng.random(len(u)) < 0.7
    u, v, w = u[keep].astype(np.uint32), v[keep].astype(np.uint32), w[keep].astype(np.uint32)
    got = ctx.graph(n, u, v, w).trials(seed=5, virtual_ranks=1, trials_per_rank=2)
    for i in range(2):
        assert int(got[0, i]) == O.mincut_trial(n, u, v, w, 5, 0, i)
    mat = np.zeros((n, n), np.uint64)
    mat[u, v] = w
    mat[v, u] = w
    assert ctx.ks_dense(mat, 5, 0, 1) == O.ks_dense(mat, 5, 0, 1)
