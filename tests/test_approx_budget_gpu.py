"""approx_cut keeps no more of a memory budget than its forest: what fitted beside that still fits after a call."""
import numpy as np
import pytest

import graphgen

pytestmark = pytest.mark.gpu


def _bytes(m):
    return 3 * ((4 * m + 255) // 256 * 256)


def test_a_graph_fits_after_an_approximate_cut(libcac):
    n, u, v, w = graphgen.erdos_renyi_m(100000, 40.0, 3, wmax=9)
    m2 = 220000
    u2, v2 = (np.random.default_rng(i).integers(0, 5000, m2).astype(np.uint32) for i in (1, 2))
    arena = 2 << 20  # 4 copies of the vertices and a count, in whole MB
    with libcac.Context(0) as c:
        g = c.graph(n, u, v, w)
        want = [(r.cut, r.level) for r in (g.approx_cut(0.9, seed=s) for s in range(3))]
    with libcac.Context(0, hbm_budget_bytes=_bytes(len(u)) + arena + _bytes(m2)) as c:
        g = c.graph(n, u, v, w)
        for s in range(3):  # (the room for the second graph holds the survivor list meanwhile)
            r = g.approx_cut(0.9, seed=s)
            assert (r.cut, r.level) == want[s]
        assert c.device_bytes == _bytes(len(u)) + arena
        g2 = c.graph(5000, u2, v2)
        assert c.device_bytes == _bytes(len(u)) + arena + _bytes(m2)
        for s in range(3):  # and without the list
            r = g.approx_cut(0.9, seed=s)
            assert (r.cut, r.level) == want[s]
        assert g2.m == m2
