"""Triangle counts through hub rows (sk_wcoj.cu) against the CPU oracle, exactly."""
import numpy as np
import pytest

import oracle as O
from strata_b200 import gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,scale", [(4096, 40_000, 0), (4096, 300_000, 0), (4097, 300_001, 0), (8192, 500_000, 0),
                                       (9000, 600_000, 0), (0, 40_003, 13), (0, 300_003, 14), (0, 1_000_003, 16)])
def test_triangle_hub_rows(engine, n, m, scale):
    # sizes around the row widths (4,096 and 8,192 labels), lists around one
    # entry per lane, labels beyond the rows; with repeats and self-loops
    import torch
    rng = np.random.default_rng(m)
    if scale:
        x, y = gen.rmat(scale, m, seed=m)
        n = 1 << scale
    else:
        x, y = (rng.integers(0, n, m).astype(np.uint32) for _ in range(2))
    hub = rng.integers(0, 40, 4000).astype(np.uint32)  # a few vertices of very high degree
    far = rng.integers(0, n, 4000).astype(np.uint32)
    x, y = np.concatenate([x, hub, far, x[:500], [7, n - 1]]), np.concatenate([y, far, hub, y[:500], [7, n - 1]])
    x, y = x.astype(np.uint32), y.astype(np.uint32)
    want = O.count_pattern(x, y)
    dx, dy = (torch.from_numpy(a.view(np.int32)).cuda() for a in (x, y))
    assert engine.count_triangle_pattern_dev(dx, dy) == want
    cuts = [0, 1, n // 3, n - 1, n + 5]
    assert sum(engine.count_triangle_pattern_range_dev(dx, dy, a, b) for a, b in zip(cuts, cuts[1:])) == want
    lo, hi = np.minimum(x, y), np.maximum(x, y)
    keep = lo != hi
    k = np.unique((lo[keep].astype(np.uint64) << np.uint64(32)) | hi[keep])
    want_u = O.count_pattern((k >> np.uint64(32)).astype(np.uint32), (k & np.uint64(0xFFFFFFFF)).astype(np.uint32))
    assert engine.count_triangles((x, y)) == want_u
    engine.set_knob(3, 2)  # the probing plan counts the same
    try:
        assert engine.count_triangle_pattern_dev(dx, dy) == want
        assert engine.count_triangles((y, x)) == want_u
    finally:
        engine.set_knob(3, 0)
