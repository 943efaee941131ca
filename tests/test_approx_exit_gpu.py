"""approx_cut in one CTA per copy: warps leave their edges as soon as the copy is one tree.

Dense graphs of few vertices and many edges, where every warp leaves in mid-list, at its own time, while others
still link; answers equal the oracle's.
"""
import numpy as np
import pytest

import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("replay", [False, True])
@pytest.mark.parametrize("n,m", [(2, 1 << 17), (3, 5000), (17, (1 << 17) - 3), (64, 1 << 17), (257, 100003), (1000, 1 << 17)])
def test_warps_leave_a_finished_copy(ctx, n, m, replay):
    rng = np.random.default_rng(n + m)
    u = rng.integers(0, n, m).astype(np.uint32)
    v = ((u + rng.integers(1, n, m)) % n).astype(np.uint32)
    w = np.ones(m, np.uint32) if replay else rng.integers(1, 6, m).astype(np.uint32)
    g = ctx.graph(n, u, v, w)
    for seed, ranks in ((0, 1), (1, 3)):
        want = (O.approx_cut_stream if replay else O.approx_cut)(n, u, v, w, 0.9, seed, ranks)
        for _ in range(5):  # the same answer whatever the warps' order
            r = g.approx_cut(0.9, seed=seed, virtual_ranks=ranks, seed_replay=replay)
            assert (r.cut, r.level) == want
