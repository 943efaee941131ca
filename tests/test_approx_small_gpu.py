"""approx_cut with a copy's forest in one CTA, and by rounds just above its limits: answers equal the oracle's."""
import numpy as np
import pytest

import graphgen
import pyoracle as O
from test_approx_rounds_gpu import _check, _edge_degree

pytestmark = pytest.mark.gpu

N, M = 16384, 1 << 17  # the one-CTA form's limits


@pytest.mark.parametrize("replay", [False, True])
@pytest.mark.parametrize("n,level,p,ranks", [
    (2, 1, 0.9, 1), (3, 1, 0.5, 2), (33, 1, 0.9, 1), (700, 3, 0.9, 3), (1025, 2, 0.995, 1), (N - 1, 1, 0.9, 2),
    (N, 1, 0.5, 1), (N + 1, 1, 0.9, 1), (20011, 1, 0.9, 3), (500, 2, 1 - 1e-10, 2),
])
def test_both_sides_of_the_vertex_limit(ctx, n, level, p, ranks, replay):
    wmax = 1 if replay else 5
    degree = min(n - 1.0, _edge_degree(n, O.approx_trials(p), level, wmax))
    _, u, v, w = graphgen.erdos_renyi_m(n, degree, 11 + n, wmax=wmax)
    _check(ctx, n, u, v, w, p, ranks, replay, range(4))


@pytest.mark.parametrize("m", [M - 1, M, M + 1])
def test_both_sides_of_the_edge_limit(ctx, m):
    n = 9000
    rng = np.random.default_rng(m)
    u, v = (rng.integers(0, n, m).astype(np.uint32) for _ in range(2))
    w = rng.integers(0, 3, m).astype(np.uint32)  # zero weights are never kept
    _check(ctx, n, u, v, w, 0.9, 2, False, range(2))


def test_many_copies_take_the_levels_in_turn(ctx):
    # 300 copies: more than the device has SMs, one level per launch
    p = 1 - np.exp(-300.5 * -np.log(1 - 0.9) / O.approx_trials(0.9))
    _, u, v, w = graphgen.erdos_renyi_m(200, 14.0, 5, wmax=9)
    _check(ctx, 200, u, v, w, min(float(p), 1 - 1e-16), 1, False, range(2))


def test_disconnected_and_more_ranks_than_edges(ctx):
    u = np.array([0, 1, 4], np.uint32)
    v = np.array([1, 2, 5], np.uint32)
    w = np.array([9, 9, 9], np.uint32)
    for ranks in (1, 2, 7):
        _check(ctx, 6, u, v, w, 0.9, ranks, False, range(2))
