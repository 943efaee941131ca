"""Queries that run out of their memory budget give back what they held, whichever allocation failed."""
import numpy as np
import pytest

import graphgen

pytestmark = pytest.mark.gpu

SCRATCH = 64 << 10  # a context keeps scratch buffers between queries, of whole multiples of this


def test_every_failing_allocation_gives_the_rest_back(libcac):
    # roots of 46 and 52 vertices, which are leaves, and 20 roots of 156, which are contracted
    gs = [graphgen.erdos_renyi_m(150, 6.7, 1, wmax=9), graphgen.erdos_renyi_m(400, 30.0, 2, wmax=9),
          graphgen.erdos_renyi_m(170, 7.6, 3, wmax=9)]
    with libcac.Context(0) as c:
        want = [r.cut for r in c.mincut_batch([c.graph(*g) for g in gs], 0.9)]
    budget, failed = sum(12 * len(g[1]) for g in gs) + (1 << 20) + 16 * 256, 0
    while True:
        with libcac.Context(0, hbm_budget_bytes=budget) as c:
            graphs = [c.graph(*g) for g in gs]
            loaded = c.device_bytes
            try:
                got = [r.cut for r in c.mincut_batch(graphs, 0.9)]
            except libcac.CacError as e:
                assert e.status == -2
                assert (c.device_bytes - loaded) % SCRATCH == 0, budget
                failed += 1
            else:
                assert got == want
                break
        budget += SCRATCH // 2
        assert budget < 64 << 20
    assert failed >= 20  # error word, Stage 1's five buffers, roots, dense descriptors, two steps' buffers


def _dense(n, m, seed):
    rng = np.random.default_rng(seed)
    iu, ju = np.triu_indices(n, 1)
    at = rng.permutation(len(iu))[:m]
    return n, iu[at].astype(np.uint32), ju[at].astype(np.uint32), rng.integers(1, 9, m).astype(np.uint32)


def test_server_out_of_budget_at_a_step_with_leaves(libcac):
    # one trial each: a root of 131 vertices (69,168 bytes) and a leaf. In the step that has both, the leaf's
    # descriptors come first; where these do not fit, the root has to be given back all the same, or the
    # leaf's query does not fit any more either. Whether both are admitted together depends on the threads' timing.
    big, leaf = _dense(135, 4225, 1), _dense(20, 40, 2)
    budget = 7 * SCRATCH - SCRATCH // 2  # a leaf alone needs seven scratch buffers
    fits = 0
    while fits < 8:
        with libcac.Server(0, budget) as s:
            gl = s.graph(*leaf)
            try:
                want = s.poll(s.submit("square_root", gl, 0.5))[0].cut
                fits += 1
            except libcac.CacError:
                want = None
        for order in (0, 1, 0, 1, 0):
            with libcac.Server(0, budget) as s:
                gb, gl = s.graph(*big), s.graph(*leaf)
                for _ in range(4):
                    tickets = [s.submit("square_root", g, 0.5) for g in ((gb, gl) if order == 0 else (gl, gb))]
                    for t in tickets:
                        try:
                            s.poll(t)
                        except libcac.CacError as e:
                            assert e.status == -2
                    if want is not None:
                        assert s.poll(s.submit("square_root", gl, 0.5))[0].cut == want
        budget += SCRATCH // 4
