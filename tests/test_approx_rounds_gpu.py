"""approx_cut by sampling rounds and survivors: every answer equals the oracle's.

The answer is the first level whose kept edges leave some copy disconnected, so one missing or one
wrong union changes it; the densities below put the break between two levels (a vertex of some copy
loses all its edges with probability about one half), and several seeds fall on both sides.
"""
import math

import numpy as np
import pytest

import graphgen
import pyoracle as O

pytestmark = pytest.mark.gpu


def _edge_degree(n, copies, level, wmax):
    """Mean degree of G(n, M) with weights 1..wmax at which `level` isolates about one vertex of copies * n."""
    q = 1 - 0.5 ** level
    g = sum(q ** w for w in range(1, wmax + 1)) / wmax
    return math.log(copies * n) / (1 - g)


def _check(ctx, n, u, v, w, p, ranks, replay, seeds):
    g = ctx.graph(n, u, v, w)
    want = [(O.approx_cut_stream if replay else O.approx_cut)(n, u, v, w, p, s, ranks) for s in seeds]
    got = [g.approx_cut(p, seed=s, virtual_ranks=ranks, seed_replay=replay) for s in seeds]
    assert [(r.cut, r.level) for r in got] == want
    return {x[1] for x in want}


@pytest.mark.parametrize("replay", [False, True])
@pytest.mark.parametrize("n,level,p,ranks", [
    (2400, 1, 0.9, 1),   # about 2^15 edges: cut to one below, then to one above the line between the two routes
    (6001, 1, 0.9, 3),   # 4 copies; n, m and the slices odd
    (5003, 2, 0.5, 2),   # 2 copies
    (4099, 2, 0.95, 5),  # 5 copies: two idle lanes per warp
    (3001, 1, 0.995, 4), # 9 copies
    (900, 2, 1 - 1e-10, 2),  # 37 copies: more than a survivor's mask holds
])
def test_levels_near_the_break(ctx, n, level, p, ranks, replay):
    copies = O.approx_trials(p)
    wmax = 1 if replay else 5
    _, u, v, w = graphgen.erdos_renyi_m(n, _edge_degree(n, copies, level, wmax), 70 + n, wmax=wmax)
    cuts = [len(u)]
    if n == 2400:
        while len(u) < (1 << 15) + 5:
            u, v, w = np.tile(u, 2), np.tile(v, 2), np.tile(w, 2)
        cuts = [(1 << 15) - 1, 1 << 15, (1 << 15) + 5]
    for m in cuts:
        _check(ctx, n, u[:m], v[:m], w[:m], p, ranks, replay, range(4))


@pytest.mark.parametrize("replay", [False, True])
def test_both_sides_of_the_break_occur(ctx, replay):
    n, wmax = 20000, 1 if replay else 42
    level = 1 if replay else 4
    _, u, v, w = graphgen.erdos_renyi_m(n, _edge_degree(n, 4, level, wmax), 5, wmax=wmax)
    assert len(_check(ctx, n, u, v, w, 0.9, 2, replay, range(8))) > 1


@pytest.mark.parametrize("order", ["sorted", "ring of cliques"])
def test_samples_without_a_giant_component(ctx, order):
    # sorted by vertex: a round sees some vertices' edges only. Cliques of 48 in a ring of heavy edges:
    # the rounds leave many large trees, so nearly every edge is a survivor, more than their list holds
    if order == "sorted":
        n, u, v, w = graphgen.erdos_renyi_m(9000, 40.0, 6, wmax=9)
        at = np.lexsort((v, u))
        u, v, w = u[at], v[at], w[at]
    else:
        k, cliques = 48, 90
        iu, ju = np.triu_indices(k, 1)
        base = np.repeat(np.arange(cliques) * k, len(iu))
        ring = np.arange(cliques) * k
        n = k * cliques
        u = np.concatenate([np.tile(iu, cliques) + base, ring]).astype(np.uint32)
        v = np.concatenate([np.tile(ju, cliques) + base, np.roll(ring, 1)]).astype(np.uint32)
        w = np.concatenate([np.full(len(base), 1), np.full(cliques, 1 << 20)]).astype(np.uint32)
    assert max(_check(ctx, n, u, v, w, 0.9, 3, False, range(3))) >= 2


def test_bitmap_larger_than_shared_memory(ctx):
    n = 1600033
    g = ctx.generate("erdos_renyi_m", seed=8, n=n, avg_degree=_edge_degree(n, 1, 1, 1), wmax=1)
    u, v, w = g.edges()
    for s in (0, 1):
        r = g.approx_cut(0.3, seed=s)
        assert (r.cut, r.level) == O.approx_cut(n, u, v, w, 0.3, s, 1)


def test_budget_without_room_for_the_survivor_list(libcac):
    import cac
    n, u, v, w = graphgen.erdos_renyi_m(30000, 30.0, 4, wmax=3)
    with cac.Context(0, hbm_budget_bytes=(12 * len(u) + 3 * 256 + (1 << 20))) as c:
        g = c.graph(n, u, v, w)
        assert c.device_bytes + 4 * n * 4 + 2 * len(u) > (12 * len(u) + 3 * 256 + (1 << 20))
        for s in (0, 1):
            r = g.approx_cut(0.9, seed=s, virtual_ranks=2)
            assert (r.cut, r.level) == O.approx_cut(n, u, v, w, 0.9, s, 2)
