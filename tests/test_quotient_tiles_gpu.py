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
