"""Contractions at the edges of their CTA sizes and row index, against the oracle's replay of the same draws."""
import numpy as np
import pytest

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
