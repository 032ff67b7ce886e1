"""Calls under a context's memory cap: a form that wants more memory gives way
to one that fits, with the uncapped result."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(n, m, seed=1):
    rng = np.random.default_rng(seed)
    s, d = rng.integers(0, n, m).astype(np.uint32), rng.integers(0, n, m).astype(np.uint32)
    return s, d, rng.integers(1, 100, m).astype(np.int64)


def _same(a, b):
    return all(np.array_equal(getattr(a, f), getattr(b, f)) for f in a.__dataclass_fields__ if f != "stats")


@pytest.mark.parametrize("n,m,cap", [(20, 40, 48 << 10), (20, 40, 128 << 10), (20, 40, 160 << 10),
                                     (200, 300, 128 << 10)])
def test_small_tropical_calls(engine, n, m, cap):
    # the input scan's own bitmap takes 128 KB; the rest of these calls far less
    from strata_b200 import Engine
    edges = _graph(n, m)
    with Engine(0, mem_cap=cap) as small:
        got = small.mssp_trop([0, 3], edges)
        assert _same(got, engine.mssp_trop([0, 3], edges))
        assert got.stats["universe"] == len(np.unique(np.concatenate([edges[0], edges[1], [0, 3]])))
        if n == 20:
            assert _same(small.shortest_paths_trop(edges), engine.shortest_paths_trop(edges))
