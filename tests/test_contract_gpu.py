"""Contractions at the edges of their CTA sizes and row index, against the oracle's replay of the same draws."""
import numpy as np
import pytest

import graphgen
import pyoracle as O

pytestmark = pytest.mark.gpu


def _weights(n, kind, seed):
    rng = np.random.default_rng(seed)
    w = np.triu(rng.integers(0, 100, (n, n)).astype(np.uint64), 1)
    if kind == "hub":  # most draws are loops after the first ones: many short batches, single-warp tails
        w[0, 1:] = rng.integers(1, 1 << 12, n - 1, dtype=np.uint64)
    elif kind == "pair":  # nearly every draw is one edge: rounds end above the target and are continued
        w[n // 3, n // 2] = np.uint64(1) << np.uint64(31)
    elif kind == "wide":  # 64-bit entries, zero columns at the end of rows
        w *= np.uint64(1 << 25)  # (below the 2^55 that a trial accepts)
        w[:, -40:] *= np.uint64(0)
        w[0, -40:] = 1
    return w + w.T


# 256 and 724 vertices: the last of 128 and 256 threads; 1024: one row per index entry, above it 2, 3 and 5
@pytest.mark.parametrize("kind", ["plain", "hub", "pair", "wide"])
@pytest.mark.parametrize("n", [129, 255, 256, 257, 723, 724, 725, 1024, 1025, 2049, 4097])
def test_trial_matches_replay(ctx, n, kind):
    mat = _weights(n, kind, n)
    assert ctx.ks_dense(mat, 3, 1, 5) == O.ks_dense(mat, 3, 1, 5)


@pytest.mark.parametrize("n", [300, 700, 1500])
def test_children_below_a_missed_target_stay_in_range(libcac, n):
    # a run planned ahead whose first children stop off their target draws, below them, from matrices and
    # prefixes that hold what earlier runs left in the memory
    for seed in range(3):
        c = libcac.Context(0)
        try:
            c.generate("erdos_renyi_m", seed=seed, n=2 * n, avg_degree=200, wmax=9).trials(seed, 1, 4)
            c.generate("watts_strogatz", seed=seed, n=3 * n, k=20, p=0.3, wmax=1 << 20).trials(seed, 1, 4)
            n, u, v, w = graphgen.complete(n, seed, wmax=1)
            w = np.asarray(w, np.uint32).copy()
            w[0] = 1 << 31  # nearly every draw
            got = c.graph(n, u, v, w).trials(seed=3, virtual_ranks=1, trials_per_rank=2)
            assert c.plan_redos() == 1
            for i in range(2):
                assert int(got[0, i]) == O.mincut_trial(n, u, v, w, 3, 0, i)
        finally:
            c.close()
