"""Connected components in one CTA, and just above its limits, on graphs with long chains, hubs and many components."""
import numpy as np
import pytest

import pyoracle as O

pytestmark = pytest.mark.gpu

SMALL_N = (64 * 1024 - 256) // 4  # the one-CTA form's vertex limit


def _shapes(n):
    i, rng = np.arange(n), np.random.default_rng(n)
    side = int(n ** 0.5)
    at = np.arange(side * side).reshape(side, side)
    clique = np.triu_indices(16, 1)
    base = np.repeat(np.arange(n // 16)[:400] * 16, 120)
    return {
        "path": (i[:-1], i[1:]),
        "path backwards": (i[:0:-1], i[-2::-1] if n > 1 else i[:0]),
        "ring": (i, (i + 1) % n),
        "ring lattice": (np.concatenate([i] * 4), np.concatenate([(i + d) % n for d in range(1, 5)])),
        "grid": (np.concatenate([at[:, :-1].ravel(), at[:-1].ravel()]), np.concatenate([at[:, 1:].ravel(), at[1:].ravel()])),
        "star at 0": (np.zeros(n - 1, np.int64), i[1:]),
        "star at the last": (np.full(n - 1, n - 1), i[:-1]),
        "hubs": (np.concatenate([np.full(n, n - 1), np.full(n, n // 2), np.zeros(n, np.int64)]),
                 np.concatenate([i % 1000 % n, i, n - 1 - i // 7])),
        "matching": (i[: n // 2 * 2: 2], i[1::2]),
        "tree": ((i[1:] * rng.random(n - 1)).astype(np.int64), i[1:]),
        "cliques": (np.tile(clique[0], len(base) // 120) + base, np.tile(clique[1], len(base) // 120) + base),
        "two paths": (i[:-2], i[2:]),
    }


@pytest.mark.parametrize("order", ["as numbered", "reversed", "relabelled"])
@pytest.mark.parametrize("n", [33, 1025, 5000, SMALL_N - 1, SMALL_N, SMALL_N + 1])
def test_labels(ctx, n, order):
    rng = np.random.default_rng(1)
    for name, (u, v) in _shapes(n).items():
        if order == "reversed":
            u, v = n - 1 - u, n - 1 - v
        elif order == "relabelled":
            q, p = rng.permutation(n), rng.permutation(len(u))
            u, v = q[u][p], q[v][p]
        u, v = u.astype(np.uint32), v.astype(np.uint32)
        want_count, want = O.cc_labels(n, u, v)
        count, lab, _ = ctx.graph(n, u, v).connected_components(seed=2, virtual_ranks=3)
        assert count == want_count and np.array_equal(lab, want), name
        lab = np.zeros(n, np.uint32)
        assert ctx.cc_edges(n, u, v, labels=lab).num_components == want_count
        assert np.array_equal(lab, want), name
