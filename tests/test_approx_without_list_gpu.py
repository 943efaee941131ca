"""approx_cut without a survivor list (more than 32 copies, or no room in the budget): answers, and that it keeps the rounds."""
import numpy as np
import pytest

import graphgen
import pyoracle as O
from test_approx_rounds_gpu import _edge_degree

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("replay", [False, True])
@pytest.mark.parametrize("n,p,ranks", [(17001, 1 - 1e-10, 2), (30011, 1 - 1e-9, 1), (50001, 0.96, 3)])
def test_answers(ctx, n, p, ranks, replay):
    # 37, 33 and 6 copies: forests with a thread per vertex and copy; the first two without a list
    wmax = 1 if replay else 3
    copies = O.approx_trials(p)
    assert copies == {17001: 37, 30011: 33, 50001: 6}[n]
    _, u, v, w = graphgen.erdos_renyi_m(n, _edge_degree(n, copies, 1, wmax), n, wmax=wmax)
    g = ctx.graph(n, u, v, w)
    for seed in (0, 1):
        r = g.approx_cut(p, seed=seed, virtual_ranks=ranks, seed_replay=replay)
        want = (O.approx_cut_stream if replay else O.approx_cut)(n, u, v, w, p, seed, ranks)
        assert (r.cut, r.level) == want


def test_time_without_room_for_the_list(libcac):
    # With the list a level takes its rounds and the few edges outside the giant components; without it the
    # rounds and a test of every quad, which on G(10^6, 15.2 M edges) is eight times 85 us, here a quarter of that:
    # less than the rounds and survivors take again. One pass of union walks from singletons is 2.4 times them.
    n, wmax = 300000, 5
    _, u, v, w = graphgen.erdos_renyi_m(n, _edge_degree(n, 4, 2, wmax), 4, wmax=wmax)
    m = len(u)
    forest = 16 * n + 4 + 256 + 16
    budget = 3 * ((4 * m + 255) // 256 * 256) + (forest + 2 * (1 << 20)) // (1 << 20) * (1 << 20)
    times = []
    for b in (0, budget):
        with libcac.Context(0, hbm_budget_bytes=b) as c:
            g = c.graph(n, u, v, w)
            r = [g.approx_cut(0.9, seed=s) for s in (0, 0, 0, 1, 2, 3, 4, 5, 6)]
            if b:
                assert c.device_bytes + m > b  # no room for the list
            times.append((float(np.median([x.device_ms / max(1, x.level) for x in r[2:]])), [(x.cut, x.level) for x in r]))
    assert times[0][1] == times[1][1]
    assert times[1][0] < 2 * times[0][0], times
