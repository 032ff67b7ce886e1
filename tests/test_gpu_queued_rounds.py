"""Direct-addressed rounds enqueued in groups: fixpoints that end at and around
a group's last round, the cap inside and at the end of a group, an error in
one of the group's rounds, and both sides of the index size from which the
rounds run one by one."""
import numpy as np
import pytest

import oracle as O
import strata_b200 as S

pytestmark = pytest.mark.gpu

I64_MAX = 2**63 - 1


@pytest.mark.parametrize("n", [1, 6, 7, 8, 9, 15, 16, 17, 40])
@pytest.mark.parametrize("wide", [False, True])
def test_chain_rounds(engine, n, wide):
    w = np.full(n, (1 << 40) if wide else 3, np.int64)
    s, d = np.arange(n), np.arange(1, n + 1)
    got = engine.shortest_paths_trop((s, d, w))
    want = O.fast_trop(0, s, d, w)
    assert np.array_equal(got.src, want[0]) and np.array_equal(got.dst, want[1]) and np.array_equal(got.w, want[2])
    assert got.stats["rounds"] == want[-1] and got.stats["plan"] == 2


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 7, 12, 13, 14, 21])
def test_negative_cycle_at_the_cap(engine, n):
    """The cap is n + 2 rounds: 3 .. 23, below, at and past a group's end."""
    s, d = np.arange(n), (np.arange(n) + 1) % n
    with pytest.raises(S.NegativeWeightCycle):
        engine.shortest_paths_trop((s, d, np.full(n, -1, np.int64)))
    with pytest.raises(S.NegativeWeightCycle):  # weights that would overflow only past the cap
        engine.shortest_paths_trop((s, d, np.full(n, -(2**62) // (n + 8), np.int64)))
    assert len(engine.shortest_paths_trop((s, d, np.full(n, 1, np.int64)))) == n * n


@pytest.mark.parametrize("at", [1, 6, 7, 8, 9, 15, 16])
def test_overflow_in_a_round_of_a_group(engine, at):
    """A chain whose sum passes i64::MAX after `at` rounds."""
    n = at + 3
    w = np.ones(n, np.int64)
    w[0], w[at] = I64_MAX - at - 1, 10
    with pytest.raises(S.TropOverflow):
        engine.mssp_trop([0], (np.arange(n), np.arange(1, n + 1), w))
    w[at] = 0
    got = engine.mssp_trop([0], (np.arange(at + 1), np.arange(1, at + 2), w[:at + 1]))
    assert len(got) == at + 1


@pytest.mark.parametrize("top", [524_287, 524_288])
def test_both_sides_of_the_queued_size(engine, top):
    # 64 sources x (top + 1) columns: 2^20 words, and two more
    rng = np.random.default_rng(top)
    s = np.concatenate([rng.integers(0, 3000, 12_000), [7, top, 2999]]).astype(np.uint32)
    d = np.concatenate([rng.integers(0, 3000, 12_000), [top, 11, 5]]).astype(np.uint32)
    w = rng.integers(1, 50, len(s)).astype(np.int64)
    src = np.arange(64, dtype=np.uint32)
    got = engine.mssp_trop(src, (s, d, w))
    cnt, fp = O.dijkstra_mssp(src, s, d, w, np.zeros(64, np.int64))
    assert len(got) == cnt and O.fingerprint(got.src, got.dst, got.w, got.inf) == fp
