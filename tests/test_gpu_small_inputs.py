"""One-block forms of small inputs: the closure kept in shared memory and the
relation sorted in one block, at the edges of their sizes, against the oracle."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns,nd,m", [(1, 1, 1), (2, 33, 5), (33, 2, 40), (31, 32, 60), (300, 300, 701), (700, 730, 2000),
                                     (760, 760, 3000), (1024, 40, 5000), (40, 1024, 5000), (1024, 1025, 300),
                                     (200, 200, 16384), (200, 200, 16385)])
def test_small_closure(engine, ns, nd, m):
    rng = np.random.default_rng(m)
    s, d = rng.integers(0, ns, m).astype(np.uint32), rng.integers(0, nd, m).astype(np.uint32)
    s[-1], d[-1] = ns - 1, nd - 1
    a, b, r = O.fast_tc(s, d)
    for plan in (0, 3, 1):
        engine.set_plan(plan)
        try:
            got = engine.transitive_closure_bool((s, d))
        finally:
            engine.set_plan(0)
        assert np.array_equal(got.src, a) and np.array_equal(got.dst, b)
        assert got.stats["rounds"] == r, plan


@pytest.mark.parametrize("m", [1, 2, 3, 31, 1023, 1024, 1025, 2047, 2048, 2049])
@pytest.mark.parametrize("wide", [False, True])
def test_small_relation(engine, m, wide):
    rng = np.random.default_rng(m)
    n = max(2, m // 3)  # repeats of the same (src, dst), some +inf
    s, d = rng.integers(0, n, m).astype(np.uint32), rng.integers(0, n, m).astype(np.uint32)
    w = rng.integers(1, (1 << 45) if wide else 90, m).astype(np.int64)
    inf = (rng.random(m) < 0.1).astype(np.uint8)
    src = rng.integers(0, n, max(1, m // 2)).astype(np.uint32)
    sw = rng.integers(0, 50, len(src)).astype(np.int64)
    got = engine.mssp_trop(src, (s, d, w, inf), source_weights=sw)
    want = O.fast_trop(1, s, d, w, inf, sources=src, source_w=sw)
    for x, y in zip((got.src, got.dst, got.w, got.inf), want):
        assert np.array_equal(x, y)
    assert got.stats["rounds"] == want[4]
    uni = len(np.unique(np.concatenate([src, s, d])))
    assert got.stats["universe"] == uni


@pytest.mark.parametrize("top", [2**20 - 1, 2**20, 2**32 - 1])
def test_distinct_ids_around_the_scan_bitmap(engine, top):
    s, d, w = np.array([0, 3, top, 3], np.uint32), np.array([3, top, 9, 9], np.uint32), np.array([1, 2, 3, 50])
    got = engine.mssp_trop([0, 3, 3], (s, d, w))
    want = O.fast_trop(1, s, d, w, sources=[0, 3, 3])
    for x, y in zip((got.src, got.dst, got.w, got.inf), want):
        assert np.array_equal(x, y)
    assert got.stats["universe"] == 4
