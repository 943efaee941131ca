"""A query that runs out of its memory budget between two levels gives back what it held."""
import pytest

import graphgen
import pyoracle as O

pytestmark = pytest.mark.gpu


def test_failed_level_releases_its_buffers(libcac):
    # K2500: 37 MB of edges and a root of 25 MB fit, the first level's children (25 MB) do not
    n, u, v, w = graphgen.erdos_renyi(150, 0.1, 4)
    want = O.exact_mincut(n, u, v, w)
    with libcac.Context(0, hbm_budget_bytes=80 << 20) as c:
        big, small = c.graph(*graphgen.complete(2500, 3)), c.graph(n, u, v, w)
        assert small.square_root(0.9, seed=2).cut == want
        held = None
        for _ in range(3):
            with pytest.raises(libcac.CacError) as e:
                big.square_root(0.9, seed=2)
            assert e.value.status == -2
            if held is not None:
                assert c.device_bytes <= held
            held = c.device_bytes
            assert small.square_root(0.9, seed=3).cut == want
