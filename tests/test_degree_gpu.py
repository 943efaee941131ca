"""The minimum weighted degree that bounds square_root's answer, on both sides of the shared-memory form's limits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# a vertex of small degree is the minimum cut: the answer is its degree, whatever the trials find
@pytest.mark.parametrize("order", ["sorted", "shuffled"])
@pytest.mark.parametrize("n,per,wmax", [(64, 63, 1), (200, 64, 9), (200, 63, 9), (3001, 65, 1 << 20), (3001, 65, 3),
                                        (40 * 1024, 64, 1), (40 * 1024 + 1, 64, 1)])
def test_bound_is_the_minimum_degree(ctx, n, per, wmax, order):
    rng = np.random.default_rng(n + per)
    m = n * per
    u = rng.integers(0, n, m)
    v = rng.integers(0, n, m)
    v = np.where(rng.random(m) < 0.05, u, v)  # loops do not count
    keep = (u != 7) & (v != 7)
    u, v = np.append(u[keep], [7] * 3), np.append(v[keep], [1, 2, 7])
    u, v = np.append(u, np.full(max(0, m - len(u)), 3)), np.append(v, np.full(max(0, m - len(v)), 4))
    w = rng.integers(1, wmax, len(u), endpoint=True)
    at = np.argsort(u, kind="stable") if order == "sorted" else rng.permutation(len(u))
    u, v, w = u[at].astype(np.uint32), v[at].astype(np.uint32), w[at].astype(np.uint32)
    deg = np.bincount(u[u != v], w[u != v], n) + np.bincount(v[u != v], w[u != v], n)
    assert ctx.graph(n, u, v, w).square_root(0.5, seed=1).cut == int(deg.min())
