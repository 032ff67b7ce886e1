"""Undirected triangle counts over ids spread widely, with and without skew,
against the CPU oracle, and the memory the counts take."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("skew", [False, True])
@pytest.mark.parametrize("m,bits", [(40_000, 18), (40_000, 22), (150_000, 24)])
def test_undirected_wide_ids(skew, m, bits):
    from strata_b200 import Engine
    rng = np.random.default_rng(bits)
    k, nodes = (m // 8, 1 << bits) if skew else (m, 1 << bits)
    a, b = ((rng.random(m) ** (3 if skew else 1) * k).astype(np.int64) for _ in range(2))
    b[:500], a[500:1000] = (a[:500] + 1) % k, b[500:1000]  # some self-loops
    a, b = np.concatenate([a, [1, 2, 0]]), np.concatenate([b, [2, 0, 1]])  # one triangle at least
    ids = rng.choice(nodes, k, replace=False).astype(np.uint32)
    ids[0] = nodes - 1
    s, d = ids[a], ids[b]
    lo, hi = np.minimum(s, d), np.maximum(s, d)
    e = np.unique((lo.astype(np.uint64) << np.uint64(32) | hi)[lo != hi])
    # the oracle's count over the vertices that occur
    _, c = np.unique(np.concatenate([e >> np.uint64(32), e & np.uint64(0xFFFFFFFF)]), return_inverse=True)
    want = O.count_pattern(c[:len(e)].astype(np.uint32), c[len(e):].astype(np.uint32))
    assert want >= 1
    with Engine(0) as eng:
        assert eng.count_triangles((s, d)) == want
        assert eng.count_triangles((d[::-1].copy(), s[::-1].copy())) == want
        if not skew and nodes > 8 * m:  # degrees and list starts, no sort of the ids
            assert eng.mem()[1] < 10 * nodes + 64 * m
