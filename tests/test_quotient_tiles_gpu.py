"""Dense Karger-Stein trials through the tile quotient, against the oracle's replay of the same draws."""
import numpy as np
import pytest

import pyoracle as O

pytestmark = pytest.mark.gpu


def _matrix(n, seed, skew, heavy):
    """Symmetric weights s_i s_j r: skewed vertex weights make groups of hundreds of members (big groups, rows
    with many members); heavy ones pass 2^32 in total (u64 entries)."""
    rng = np.random.default_rng(seed)
    s = np.ones(n) if not skew else rng.pareto(0.7, n) + 1
    s = np.minimum(s, 400.0)
    w = np.triu(np.floor(np.outer(s, s) * rng.random((n, n)) * 3).astype(np.uint64), 1)
    if heavy:
        w *= np.uint64(1 << 13)
    return w + w.T


@pytest.mark.parametrize("heavy", [False, True])
@pytest.mark.parametrize("skew", [False, True])
@pytest.mark.parametrize("n", [129, 131, 182, 257, 361, 363, 512, 731, 1027, 1450])
def test_trials_match_replay(ctx, n, skew, heavy):
    # children of 8, 16 and 32 column blocks and of odd sizes; 8, 4, 2 and 1 tiles at a time
    mat = _matrix(n, n, skew, heavy)
    for trial in (0, 1):
        assert ctx.ks_dense(mat, 7, 2, trial) == O.ks_dense(mat, 7, 2, trial)


@pytest.mark.parametrize("kind", [0, 1, 2])
def test_rule_and_forced_kernels_agree_at_the_line(libcac, kind):
    import cac
    for n in (2900, 2901):
        mat = _matrix(n, n, True, False)
        with cac.Context(0) as c:
            c.set_quotient_kernel(kind)
            assert c.ks_dense(mat, 1, 0, 0) == O.ks_dense(mat, 1, 0, 0)


def test_batch_of_uneven_sizes_matches_single_queries(ctx):
    gs = [ctx.generate("erdos_renyi_m", seed=i, n=int(n), avg_degree=d, wmax=w) for i, (n, d, w) in enumerate(
        [(150, 30, 9), (700, 60, 100), (1300, 64, 3), (131, 100, 1 << 30), (400, 12, 7), (2000, 40, 1 << 31)])]
    want = [g.square_root(0.9, seed=i).cut for i, g in enumerate(gs)]
    assert [r.cut for r in ctx.mincut_batch(gs, 0.9, seeds=list(range(len(gs))))] == want


# the triangle kernel's range: children of 129 vertices to 192 (u32 entries) or 136 (u64), and just above
@pytest.mark.parametrize("heavy", [False, True])
@pytest.mark.parametrize("skew", [False, True])
@pytest.mark.parametrize("n", [180, 181, 190, 191, 226, 227, 255, 256, 269, 270, 271, 272, 385])
def test_small_children_match_replay_and_tiles(libcac, n, skew, heavy):
    import cac
    mat = _matrix(n, n, skew, heavy)
    if heavy:
        mat *= np.uint64(16)
    want = O.ks_dense(mat, 9, 0, 0)
    for kind in (0, 1):
        with cac.Context(0) as c:
            c.set_quotient_kernel(kind)
            assert c.ks_dense(mat, 9, 0, 0) == want
    u, v = np.triu_indices(n, 1)  # planned ahead
    w = np.minimum(mat[u, v], np.uint64((1 << 32) - 1)).astype(np.uint32)
    keep = w > 0
    u, v, w = u[keep].astype(np.uint32), v[keep].astype(np.uint32), w[keep]
    with cac.Context(0) as c:
        got = c.graph(n, u, v, w).trials(seed=4, virtual_ranks=1, trials_per_rank=2)
    for i in range(2):
        assert int(got[0, i]) == O.mincut_trial(n, u, v, w, 4, 0, i)
