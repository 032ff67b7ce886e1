"""Bit-row rounds at the edges of their word blocks, strips and edge windows,
against the SCC oracle (counts, fingerprints) and the restated rounds."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 129, 2048, 2049, 4096, 4097, 8300])
@pytest.mark.parametrize("mode", [0, 1])
def test_bit_row_blocks(engine, n, mode):
    # a sparse graph with one row of n/3 edges (many windows), one of exactly
    # 32 and one of 33, a long chain (many sparse rounds), repeats and a loop
    rng = np.random.default_rng(n)
    u, v = rng.integers(0, n, n).astype(np.uint32), rng.integers(0, n, n).astype(np.uint32)
    chain = np.arange(max(0, min(n - 1, 60)), dtype=np.uint32)
    parts_u, parts_v = [u, chain, u[:5]], [v, chain + 1, v[:5]]
    for row, deg in ((0, n // 3), (n // 2, 32), (n - 1, 33)):
        parts_u.append(np.full(deg, row, np.uint32))
        parts_v.append(rng.integers(0, n, deg).astype(np.uint32))
    u, v = np.concatenate(parts_u), np.concatenate(parts_v)
    nodes, off = np.array([n, 3, n], np.uint32), np.array([0, len(u), len(u) + 2, 2 * len(u) + 2], np.uint64)
    src, dst = np.concatenate([u, [0, 1], u]).astype(np.uint32), np.concatenate([v, [1, 2], v]).astype(np.uint32)
    res = engine.tc_bool_batch(nodes, off, src, dst, mode=mode)
    counts, fps = O.closure_batch(nodes, off, src, dst, threads=4)
    assert np.array_equal(res.counts, counts) and np.array_equal(res.fps, fps)
    _, _, r = O.fast_tc(u, v)
    assert res.rounds.tolist() == [r, 2, r]
