"""Several threads, each with its own context, in the kernels whose shared memory
depends on the input: one thread's size must not take another's away."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(workers):
    bad = []

    def loop(work):
        try:
            work()
        except Exception as e:  # reported by the test's own thread
            bad.append(repr(e))
    ts = [threading.Thread(target=loop, args=(w,)) for w in workers]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad, bad[:2]


def _graph(n, m, seed):
    rng = np.random.default_rng(seed)
    s, d = rng.integers(0, n, m).astype(np.uint32), rng.integers(0, n, m).astype(np.uint32)
    s[-1] = d[-1] = n - 1
    return s, d


@pytest.mark.parametrize("call,sizes", [("transitive_closure_bool", [(40, 60), (700, 900), (300, 400)]),
                                        ("count_4cliques", [(60, 300), (4000, 9000), (1500, 300_000)]),
                                        ("shortest_paths_trop", [(1_060_000, 2100), (1_300_000, 2100), (1_200_000, 2100)])])
def test_sizes_of_other_threads(engine, call, sizes):
    from strata_b200 import Engine
    inputs = []
    for i, (n, m) in enumerate(sizes):
        e = _graph(n, m, i)
        if call == "shortest_paths_trop":  # a tree: few pairs; ids past 2^20 are marked in shared memory
            e = (np.arange(1, m + 1, dtype=np.uint32) // 4 % n, np.arange(1, m + 1, dtype=np.uint32) % n,
                 np.ones(m, np.int64))
            e[1][-1] = n - 1
        inputs.append(e)
    want = [getattr(engine, call)(e) for e in inputs]

    def worker(e, w):
        def work():
            with Engine(0) as eng:
                for _ in range(150):
                    got = getattr(eng, call)(e)
                    assert got == w if isinstance(w, int) else np.array_equal(got.src, w.src)
        return work
    _run([worker(e, w) for e, w in zip(inputs, want)] * 2)


def test_circuit_sets_of_other_threads(engine):
    import torch
    from strata_b200 import Engine
    rng = np.random.default_rng(1)
    p = torch.from_numpy(rng.uniform(0.1, 0.9, 64).astype(np.float32)).cuda()
    sets = [[[[1, 2]]] * 50, [[sorted(rng.choice(np.arange(1, 65), 4, replace=False).tolist()) for _ in range(k)]
                              for k in (7, 8, 9)] * 10]
    want = []
    for q in sets:
        c = engine.compile_circuits(q, 64)
        want.append(c.forward(p).cpu())
        c.free()

    def worker(q, w):
        def work():
            with Engine(0) as eng, torch.cuda.stream(torch.cuda.Stream()) as _:
                c = eng.compile_circuits(q, 64)
                seed = torch.ones(len(q), device="cuda")
                for _ in range(300):
                    out = c.forward(p)
                    c.vjp(p, seed)
                torch.cuda.current_stream().synchronize()
                assert torch.equal(out.cpu(), w)
                c.free()
        return work
    torch.cuda.synchronize()
    _run([worker(q, w) for q, w in zip(sets, want)] * 2)
