"""The circuit compiler on both sides of its mask widths (64, 128 and 256
variables, then ordered lists) against the oracle: node counts and
bit-identical FP64 values."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
from strata_b200 import _lib as L
from strata_b200.gpu import CircuitParts, ProofSets


@pytest.mark.parametrize("n_vars", [1, 2, 63, 64, 65, 127, 128, 129, 255, 256, 257, 300])
@pytest.mark.parametrize("signed", [False, True])
def test_widths(n_vars, signed):
    lib = L.load()
    rng = np.random.default_rng(n_vars)
    probs = rng.uniform(0.05, 0.95, 1000)
    ids = np.sort(rng.choice(np.arange(1, 1001), n_vars, replace=False))
    # proofs that together hold every variable, overlapping in a few of them;
    # one repeated, one absorbed, one contradictory when signs are drawn
    cut = np.array_split(ids, max(1, n_vars // 32))
    q = []
    for part in cut:
        extra = rng.choice(ids, min(3, n_vars), replace=False)
        p = np.unique(np.concatenate([part, extra]))
        sign = np.where(signed & (rng.random(len(p)) < 0.3), -1, 1)
        q.append([int(x) for x in p * sign])
    q += [list(q[0]), sorted(set(q[-1]) | {int(ids[0])})]
    if signed:
        q.append([int(ids[0]), -int(ids[0])])
    ps = ProofSets.from_lists([q, q[:1], [], [[]]])
    out = C.c_void_p()
    rc = lib.strata_circuits_compile_host(len(ps), ps.proof_off.ctypes.data_as(C.POINTER(C.c_uint64)),
                                          ps.lit_off.ctypes.data_as(C.POINTER(C.c_uint64)),
                                          ps.lits.ctypes.data_as(C.POINTER(C.c_int64)), 1000, 0, C.byref(out))
    assert rc == 0
    parts = CircuitParts(lib, out, len(ps))
    got, nodes = parts.eval64(probs), 0
    for i, query in enumerate([q, q[:1], [], [[]]]):
        want, _, nn = O.compile_grad([sorted(p) for p in query], probs)
        assert got[i] == want
        nodes += nn
    assert parts.shape()[0] == nodes
    parts.free()
