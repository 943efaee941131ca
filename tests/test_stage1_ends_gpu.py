"""Stage 1 of square_root where the last warps hold few edges: trials against the oracle's replay."""
import numpy as np
import pytest

import pyoracle as O

pytestmark = pytest.mark.gpu


def _edges(n, m, seed):
    rng = np.random.default_rng(seed)
    u = rng.integers(0, n, m)
    v = (u + rng.integers(1, n, m)) % n
    return u.astype(np.uint32), v.astype(np.uint32), rng.integers(1, 43, m).astype(np.uint32)


# A trial's warps (32 of them, 16 when trials are many) own whole segments of 32 edges. 24,850: 800 edges a warp, the
# last one has 50, within the last 128-edge step of the one before. 24,801, 24,896, 25,600: 1, 96 and 800 of its own.
@pytest.mark.parametrize("m", [24801, 24850, 24896, 25600, 12050, 65570])
@pytest.mark.parametrize("trials", [2, 160])
def test_trials_match_replay(ctx, m, trials):
    n = 900
    u, v, w = _edges(n, m, m)
    got = ctx.graph(n, u, v, w).trials(seed=5, virtual_ranks=1, trials_per_rank=trials)
    for i in (0, 1) if trials == 2 else (0, 77, 159):
        assert int(got[0, i]) == O.mincut_trial(n, u, v, w, 5, 0, i)
