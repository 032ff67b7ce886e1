"""Circuit values and gradients on both sides of the shared-memory form's sizes:
one larger circuit among many small ones, against the FP64 oracle."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

N = 400


def _pairs(k, seed=3):
    """k overlapping pairs: the decision nodes grow with the overlap."""
    v = np.random.default_rng(seed).permutation(N)[:48] + 1
    return [sorted((int(v[i]), int(v[(i * 7 + 3) % 48]))) for i in range(k) if v[i] != v[(i * 7 + 3) % 48]]


# queries, pairs of the large one, and whether the set is staged
@pytest.mark.parametrize("nq,k,form", [(200, 4, True), (200, 16, True), (149, 17, True), (148, 18, True), (149, 18, False),
                                       (200, 19, False), (100, 19, None), (100, 22, False), (1, 18, True), (1, 22, False)])
def test_one_large_circuit(engine, nq, k, form):
    import torch
    rng = np.random.default_rng(k)
    queries = [[sorted(set(rng.integers(1, N + 1, 4).tolist())) for _ in range(3)] for _ in range(nq - 1)]
    queries.insert(nq // 2, _pairs(k))
    circ = engine.compile_circuits(queries, N)
    big = engine.compile_circuits([_pairs(k)], N)
    nodes = big.shape()[0]
    big.free()
    limit = (226 if nq <= 148 else 112) << 10
    sure = True if 20 * nodes <= limit else False if 17 * nodes > limit else None  # 17 bytes a node, 2 a child
    assert form is None or sure is None or form == sure, nodes
    p32 = rng.uniform(0.05, 0.95, N).astype(np.float32)
    p = torch.from_numpy(p32).cuda()
    P = circ.forward(p, out64=True).cpu().numpy()
    seed = rng.uniform(-1, 1, nq).astype(np.float32)
    ds = torch.from_numpy(seed).cuda()
    before = engine.launches()
    g32, g64 = circ.vjp(p, ds)
    if sure is not None:  # staged: one kernel and the FP32 copy; else values, adjoints and the copy
        assert engine.launches() - before == (2 if sure else 3), nodes
    want = np.zeros(N)
    for i, q in enumerate(queries):
        w, g, _ = O.compile_grad(q, p32.astype(np.float64))
        assert abs(P[i] - w) <= 1e-6 * max(w, 1e-30) + 1e-30
        want[:len(g)] += float(seed[i]) * np.asarray(g)
    assert np.linalg.norm(g64.cpu().numpy() - want) <= 1e-5 * np.linalg.norm(want)
    assert torch.equal(g32, g64.float())
    circ.free()
