"""Circuit kernels on both sides of the shared-memory form's size: a set of
small circuits, one with a large circuit among them, and empty and constant
ones, against the FP64 oracle."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("big", [False, True])
def test_values_and_gradients(engine, big):
    import torch
    rng = np.random.default_rng(3)
    n = 400
    queries = [[], [[]], [[1]], [[-1]], [[5, 7], [7, 9]]]
    for _ in range(60):
        base = rng.integers(1, n + 1, 6).tolist()
        queries.append([sorted(set(base[:a] + rng.integers(1, n + 1, 2).tolist())) for a in range(1, 6)])
    if big:  # disjoint pairs: thousands of decision nodes
        v = rng.permutation(n)[:48] + 1
        queries.append([sorted((int(v[i]), int(v[(i * 7 + 3) % 48]))) for i in range(0, 30) if v[i] != v[(i * 7 + 3) % 48]])
    circ = engine.compile_circuits(queries, n)
    p32 = rng.uniform(0.05, 0.95, n).astype(np.float32)
    p = torch.from_numpy(p32).cuda()
    P, G = circ.forward(p, out64=True).cpu().numpy(), circ.grads(p).cpu().numpy()
    seed = rng.uniform(-1, 1, len(queries)).astype(np.float32)
    g64 = circ.vjp(p, torch.from_numpy(seed).cuda())[1].cpu().numpy()
    want_g = np.zeros(n)
    for i, q in enumerate(queries):
        w, g, nodes = O.compile_grad(q, p32.astype(np.float64))
        row = np.zeros(n)
        row[:len(g)] = g
        assert abs(P[i] - w) <= 1e-6 * max(w, 1e-30) + 1e-30
        assert np.linalg.norm(G[i] - row) <= 1e-5 * np.linalg.norm(row) + 1e-30
        want_g += float(seed[i]) * row
    assert np.linalg.norm(g64 - want_g) <= 1e-5 * np.linalg.norm(want_g)
    assert (max(O.compile_grad(q, p32.astype(np.float64))[2] for q in queries) > 1536) == big
    circ.free()
