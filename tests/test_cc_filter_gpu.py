"""The edge filter above 1.57 M vertices: quads of the giant component in shared memory, or the bitmap's first part."""
import numpy as np
import pytest

import graphgen
import pyoracle as O

pytestmark = pytest.mark.gpu

LINE = 32 * 48 * 1024  # vertices whose bitmap fits


def _check(ctx, n, u, v):
    want_count, want = O.cc_labels(n, u, v)
    g = ctx.graph(n, u, v)
    count, lab, _ = g.connected_components(seed=1, virtual_ranks=3)
    assert count == want_count and np.array_equal(lab, want)
    lab = np.zeros(n, np.uint32)
    assert ctx.cc_edges(n, u, v, seed=2, labels=lab).num_components == want_count
    assert np.array_equal(lab, want)


# a little above the line, ragged words and quads, above the quads' reach (6.3 M); the giant covers nearly all of
# the vertices, about half of them at random (the quads find few), or only one id in a run
@pytest.mark.parametrize("n", [LINE, LINE + 1, LINE + 131, 2000003, 4 * LINE + 77])
@pytest.mark.parametrize("kind", ["dense", "thin", "strided", "block"])
def test_labels_above_the_line(ctx, n, kind):
    rng = np.random.default_rng(n)
    m = {"dense": 4 * n, "thin": int(0.72 * n), "strided": n, "block": n}[kind]
    u, v = (rng.integers(0, n, m) for _ in range(2))
    if kind == "strided":  # every fifth id
        u, v = u // 5 * 5, v // 5 * 5
    elif kind == "block":  # ids at the end only
        u, v = n - 1 - u // 3, n - 1 - v // 3
    _check(ctx, n, u.astype(np.uint32), v.astype(np.uint32))


def test_rmat_22(ctx):
    n, u, v, _ = graphgen.rmat(22, 4, 3)
    _check(ctx, n, u, v)


def test_budget_without_room_for_the_quads(libcac):
    import cac
    n, m = LINE + 40001, 3 << 20
    rng = np.random.default_rng(3)
    u, v = (rng.integers(0, n, m).astype(np.uint32) for _ in range(2))
    want_count, want = O.cc_labels(n, u, v)
    with cac.Context(0) as c:
        c.graph(n, u, v).connected_components(seed=1)
        full = c.device_bytes
    answered = 0
    for budget in range(full - (2 << 20), full + (64 << 20), 1 << 18):  # from the first that suffices
        with cac.Context(0, hbm_budget_bytes=budget) as c:
            try:
                count, lab, _ = c.graph(n, u, v).connected_components(seed=1)
            except cac.CacError:
                assert not answered
                continue
            answered += 1
            assert count == want_count and np.array_equal(lab, want)
        if answered == 8:
            break
    assert answered
