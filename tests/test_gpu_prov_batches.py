"""Prov_k rounds that skip batches: proof sets and rounds equal the capture's
restatement where sets are full and often unchanged (dense graphs, long
cycles), where weights tie, vanish or are 1, and where they are no
probabilities at all."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _probs(kind, rng, m):
    if kind == "beta":
        return rng.beta(2.0, 5.0, m)
    if kind == "ties":
        return rng.choice([0.5, 0.25], m)
    if kind == "tiny":
        return rng.choice([1e-100, 1e-40, 1e-3, 0.9], m)
    return rng.choice([1.25, 0.5, 0.7], m)  # not probabilities


@pytest.mark.parametrize("kind", ["beta", "ties", "tiny", "other"])
@pytest.mark.parametrize("n,deg,k", [(12, 4, 8), (40, 3, 8), (60, 4, 3), (150, 2, 1), (300, 3, 8)])
def test_sets_and_rounds(engine, kind, n, deg, k):
    if kind in ("tiny", "other"):
        # sparse: where weights tie at 0 or grow with length, pruning on a
        # dense graph may never settle; fewer than 32 edges keep proofs short
        n, deg = 10 + k, 1.5
    rng = np.random.default_rng(n * 10 + k)
    m = int(n * deg)
    key = rng.permutation(n * n)
    key = key[key // n != key % n][:m]
    s, d = (key // n).astype(np.uint32), (key % n).astype(np.uint32)
    p = _probs(kind, rng, len(s)).astype(np.float64)
    qs, qt = rng.integers(0, n, 24).astype(np.uint32), rng.integers(0, n, 24).astype(np.uint32)
    got = engine.prov_capture(n, s, d, p, qs, qt, k=k)
    want, rounds = O.prov_tc(n, s, d, p, k, qs, qt)
    assert got.as_lists() == want
    assert got.target_rounds.tolist() == [rounds[t] for t in sorted(rounds)]
