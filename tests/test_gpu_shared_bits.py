"""Relations whose ids share bits: only the bits that differ are sorted, and the
results are those of the same graph over small ids."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

M = 30_000


def _edges(case):
    rng = np.random.default_rng(7)
    if case == "star":  # one source
        return np.full(M, 70_000), rng.permutation(1 << 16)[:M]
    if case == "shared":  # 12 bits of 27 differ in each column
        return (1 << 26) + rng.integers(0, 4096, M), (1 << 26) + 4096 + rng.integers(0, 4096, M)
    if case == "holes":  # bits 3..5, 11..13 and 20..23
        def take():
            return sum(rng.integers(0, 1 << w, M) << s for s, w in ((3, 3), (11, 3), (20, 4)))
        return take() | 1 << 25, take() | 1 << 24
    return np.full(M, 9), np.full(M, 9)  # one row


# sort passes of eight bits: (x, y) for the relation, (y, x) for the edges
@pytest.mark.parametrize("case,passes", [("star", 2 + 2), ("shared", 3 + 3), ("holes", 3 + 3), ("one", 0)])
def test_sort_passes(case, passes):
    from strata_b200 import Engine
    s, d = (c.astype(np.uint32) for c in _edges(case))
    w = np.random.default_rng(1).integers(1, 1000, M).astype(np.int64)
    with Engine(0, profiling=True) as eng:
        eng.set_plan(1)
        eng.reset_kernel_stats()
        got = eng.shortest_paths_trop((s, d, w))  # at most one derived pair a round: no sorts of those
        assert eng.kernel_stats()["k_onesweep"][0] == passes
        want = O.fast_trop(0, s, d, w)
        for a, b in zip((got.src, got.dst, got.w, got.inf), want):
            assert np.array_equal(a, b)
        b = eng.transitive_closure_bool((s, d))
        assert np.array_equal(b.src, got.src) and np.array_equal(b.dst, got.dst)
        m = eng.mssp_trop(s[:1], (s, d, w))
        want = O.fast_trop(1, s, d, w, sources=s[:1])
        for a, b in zip((m.src, m.dst, m.w, m.inf), want):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("m", [3_000, 30_000])
@pytest.mark.parametrize("loops", [False, True])
@pytest.mark.parametrize("base,step", [(1 << 26, 1), (0, 64), ((1 << 26) - 64, 512)])
def test_patterns(engine, m, loops, base, step):
    # the counts over ids base + step * i are those over i
    rng = np.random.default_rng(m)
    a, b = rng.integers(0, 1 << 9, m), rng.integers(0, 1 << 9, m)
    if not loops:
        a, b = a[a != b], b[a != b]
    small = (a.astype(np.uint32), b.astype(np.uint32))
    wide = ((base + step * a).astype(np.uint32), (base + step * b).astype(np.uint32))
    assert engine.count_triangle_pattern(wide) == O.count_pattern(*small)
    for fn in (engine.count_triangles, engine.count_4cliques, engine.binary_plan_intermediate):
        assert fn(wide) == fn(small), fn
