"""Connected components above 1.57 M vertices: the quads of the filter take no scratch of their own."""
import numpy as np
import pytest

import pyoracle as O

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _up(x, a=256):
    return (x + a - 1) // a * a


def _scratch(n, m):
    """Parents, tile counts and offsets, totals, one rank, bitmap, regions, survivors, draws (one rank)."""
    tiles, words = (n + 1023) // 1024, (n + 31) // 32
    draws = int(np.float32(n) ** np.float32(1.045) * np.float32(1.2))
    assert draws < m
    return (_up(4 * n) + 2 * _up(4 * tiles + 4) + 256 + 256 + _up(4 * words + 4) + _up(4096) + _up((m + 4096) * 8) +
            _up((1 + (draws + 31) // 32) * 8))


def test_scratch_is_what_the_query_needs_without_them(libcac):
    m = 5000000
    # a size whose scratch ends within the quads' bytes (n / 32) of the next whole MB
    n = next(n for n in range(1600003, 2000000, 1009) if 4096 < -_scratch(n, m) % MB < n // 32 - 4096)
    arena = _up(_scratch(n, m), MB)
    with libcac.Context(0) as c:
        g = c.generate("erdos_renyi_m", seed=3, n=n, avg_degree=2 * m / n, wmax=1)
        assert g.m == m
        u, v, _ = g.edges()
    want_count, want = O.cc_labels(n, u, v)
    graph, second = 3 * _up(4 * m), 80000  # the second graph: just below 1 MB
    labels, labels_bytes = np.zeros(n, np.uint32), _up(4 * n + 4, MB)
    with libcac.Context(0, hbm_budget_bytes=graph + arena + labels_bytes + MB) as c:
        g = c.graph(n, u, v)
        for seed in (0, 0, 0, 1):  # direct, captured, replayed
            count, labels, _ = g.connected_components(seed=seed, virtual_ranks=1)
            assert count == want_count and np.array_equal(labels, want)
        assert c.device_bytes == graph + arena + labels_bytes
        c.graph(1000, u[:second] % 1000, v[:second] % 1000)


@pytest.mark.parametrize("labels", [False, True])
def test_edges_from_the_host(libcac, labels):
    n, m = 1700021, 6000000
    rng = np.random.default_rng(4)
    u, v = (rng.integers(0, n, m).astype(np.uint32) for _ in range(2))
    want_count, want = O.cc_labels(n, u, v)
    with libcac.Context(0) as c:
        for _ in range(3):
            lab = np.zeros(n, np.uint32)
            r = c.cc_edges(n, u, v, labels=lab if labels else None)
            assert r.num_components == want_count
            assert not labels or np.array_equal(lab, want)
