"""Calls under a context's memory cap: a form that wants more memory gives way
to one that fits, with the uncapped result."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(n, m, seed=1):
    rng = np.random.default_rng(seed)
    s, d = rng.integers(0, n, m).astype(np.uint32), rng.integers(0, n, m).astype(np.uint32)
    return s, d, rng.integers(1, 100, m).astype(np.int64)


def _same(a, b):
    return all(np.array_equal(getattr(a, f), getattr(b, f)) for f in a.__dataclass_fields__ if f != "stats")


@pytest.mark.parametrize("n,m,cap", [(20, 40, 48 << 10), (20, 40, 128 << 10), (20, 40, 160 << 10),
                                     (200, 300, 128 << 10)])
def test_small_tropical_calls(engine, n, m, cap):
    # the input scan's own bitmap takes 128 KB; the rest of these calls far less
    from strata_b200 import Engine
    edges = _graph(n, m)
    with Engine(0, mem_cap=cap) as small:
        got = small.mssp_trop([0, 3], edges)
        assert _same(got, engine.mssp_trop([0, 3], edges))
        assert got.stats["universe"] == len(np.unique(np.concatenate([edges[0], edges[1], [0, 3]])))
        if n == 20:
            assert _same(small.shortest_paths_trop(edges), engine.shortest_paths_trop(edges))


def test_compiled_circuits():
    # per node a kind, two words and three floats; per child and level a word;
    # per query two first entries and a root of 4 bytes and a 64-bit level start
    import torch
    from strata_b200 import Engine
    nq = 1023

    def cls(b):  # size classes of the context's blocks
        step = 256 if b <= 1 << 20 else 1 << (b.bit_length() - 4)
        return -(-b // step) * step
    with Engine(0) as eng:
        one = eng.compile_circuits([[[1, 2], [2, 3]]], 3)
        nodes, levels = one.shape()
        assert nodes == 19  # three decisions of five nodes, four constants
        one.free()
        held = eng.mem()[0]
        circ = eng.compile_circuits([[[1, 2], [2, 3]]] * nq, 3)
        assert eng.mem()[0] - held <= (cls(nq * nodes) + 5 * cls(4 * nq * nodes) + cls(4 * nq * 18) + cls(8 * (nq + 1)) +
                                       cls(4 * nq) + cls(8 * (nq + 1)) + cls(4 * nq * (levels + 1)))
        p = torch.full((3,), 0.5, device="cuda")
        assert torch.equal(circ.forward(p), torch.full((nq,), 0.375, device="cuda"))
        circ.free()


def test_closure_gives_way_to_the_tuple_plan(engine):
    # 4,500 disjoint edges of 9,000 nodes: bit rows of 31 MB for a relation of 36 KB
    from strata_b200 import Engine
    n = 9000
    s = np.arange(0, n, 2, dtype=np.uint32)
    want = engine.transitive_closure_bool((s, s + 1))
    assert np.array_equal(want.src, s) and np.array_equal(want.dst, s + 1)
    mats = 3 * (n - 1) * -(-n // 128) * 16
    for cap in [mats // 2] + [int(mats * f) for f in (1.005, 1.01, 1.05, 1.1, 1.15, 1.3)]:
        with Engine(0, mem_cap=cap) as small:
            small.set_plan(1)
            assert _same(small.transitive_closure_bool((s, s + 1)), want)
        with Engine(0, mem_cap=cap) as small:
            assert _same(small.transitive_closure_bool((s, s + 1)), want), cap


def _calls():
    s, d, w = _graph(2500, 2700)  # queued rounds: heads for 2,500 * 79 words
    t = _graph(700, 2000, 2)
    rng = np.random.default_rng(4)
    hub = tuple((rng.random(60_000) ** 3 * 3000).astype(np.uint32) for _ in range(2))  # hub rows from 2^15 edges on
    small = _graph(300, 700, 5)[:2]  # one-block closure
    rows = _graph(3000, 5000, 6)[:2]
    return {"sparse paths": lambda e: e.shortest_paths_trop((s, d, w)), "paths": lambda e: e.shortest_paths_trop(t),
            "mssp": lambda e: e.mssp_trop([1, 2, 3], (s, d, w)), "small closure": lambda e: e.transitive_closure_bool(small),
            "closure": lambda e: e.transitive_closure_bool(rows), "triangles": lambda e: e.count_triangles(hub)}


@pytest.mark.parametrize("name", list(_calls()))
def test_more_memory_never_fails(engine, name):
    # a form chosen because its estimate fits, and that then does not, would
    # fail above a cap at which a smaller form ran
    from strata_b200 import Engine
    from strata_b200.gpu import OutOfMemory
    call = _calls()[name]
    want = call(engine)
    with Engine(0) as eng:
        call(eng)
        peak = eng.mem()[1]
    ran = False
    for cap in np.geomspace(peak / 40, peak * 1.1, 60).astype(int).tolist() + [peak]:
        with Engine(0, mem_cap=cap) as eng:
            try:
                got = call(eng)
            except OutOfMemory:
                assert not ran, (cap, peak)
                continue
            ran = True
            assert got == want if isinstance(want, int) else _same(got, want)
    assert ran
