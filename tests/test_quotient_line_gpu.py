"""The line between tiles and rows of the quotient with u64 entries: forced kernels and the rule agree, and the replay."""
import numpy as np
import pytest

import pyoracle as O
from test_quotient_tiles_gpu import _matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("skew", [False, True])
@pytest.mark.parametrize("n", [2901, 3607, 5000, 5001])
def test_rule_agrees_with_rows(libcac, n, skew):
    mat = _matrix(n, n, skew, True) * np.uint64(8)
    assert int(mat.sum()) // 2 >= 1 << 32
    got = []
    for kind in (0, 1, 2):
        with libcac.Context(0) as c:
            c.set_quotient_kernel(kind)
            got.append([c.ks_dense(mat, 5, 1, t) for t in (0, 1)])
    assert got[0] == got[1] == got[2]
    if n == 2901:
        assert got[0] == [O.ks_dense(mat, 5, 1, t) for t in (0, 1)]


def test_trials_match_replay_above_the_line_of_narrow_entries(ctx):
    n = 3001
    rng = np.random.default_rng(3)
    u, v = np.triu_indices(n, 1)
    w = rng.integers(1, 1 << 31, len(u)).astype(np.uint32)
    got = ctx.graph(n, u.astype(np.uint32), v.astype(np.uint32), w).karger_stein_trials(seed=2, trials=2)
    assert [int(x) for x in got] == [O.ks_trial(n, u.astype(np.uint32), v.astype(np.uint32), w, 2, i) for i in range(2)]
