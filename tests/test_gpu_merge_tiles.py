"""The one-pass merge at its tiles' edges and over many tiles (each learns the
rows before it from its predecessors): the combine with Δ', Δ' alone, and the
minimum merged in place, against dictionaries."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

INF = 2**63 - 1


def _t(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a).view({4: np.int32, 8: np.int64}[a.dtype.itemsize])).cuda()


@pytest.mark.parametrize("kb", [4, 8])
@pytest.mark.parametrize("na,nb", [(1023, 1024), (1024, 1024), (1025, 1024), (2047, 1), (1, 2048), (2049, 2049),
                                   (400_000, 3), (5, 400_000), (250_000, 250_001)])
def test_tiles(engine, kb, na, nb):
    import torch
    kt = {4: np.uint32, 8: np.uint64}[kb]
    rng = np.random.default_rng(na + nb)
    for spread in (1, 4):  # mostly equal pairs, then few
        a, b = (np.sort(rng.permutation(max(na, nb) * spread + 1)[:n]).astype(kt) for n in (na, nb))
        aw, bw = rng.integers(0, 4, na), rng.integers(0, 4, nb)
        aw[rng.random(na) < 0.1] = INF
        hit = np.isin(b, a)
        at = np.searchsorted(a, b).clip(0, na - 1)
        better = ~hit | (bw < aw[at])
        keys = np.union1d(a, b)
        w = np.full(len(keys), INF)
        np.minimum.at(w, np.searchsorted(keys, a), aw)
        np.minimum.at(w, np.searchsorted(keys, b), bw)
        ka, kb_, wa, wb = _t(a), _t(b), _t(aw), _t(bw)
        fo, do = (torch.empty(n, dtype=ka.dtype, device="cuda") for n in (na + nb, nb))
        fw, dw = (torch.empty(n, dtype=torch.int64, device="cuda") for n in (na + nb, nb))
        nf, nd = C.c_uint64(), C.c_uint64()
        p = lambda t: t.data_ptr()
        lib, chk, ctx = engine.lib, engine._check, engine.ctx
        got = lambda t, n, dt: t[:n].cpu().numpy().view(dt)
        for trop in (False, True):
            x = (p(wa), p(wb), p(fw), p(dw)) if trop else (None,) * 4
            chk(lib.strata_op_merge_diff(ctx, kb, p(ka), x[0], na, p(kb_), x[1], nb, p(fo), x[2], p(do), x[3],
                                         C.byref(nf), C.byref(nd)))
            new = better if trop else ~hit
            assert np.array_equal(got(fo, nf.value, kt), keys) and np.array_equal(got(do, nd.value, kt), b[new])
            if trop:
                assert np.array_equal(got(fw, nf.value, np.int64), w)
                assert np.array_equal(got(dw, nd.value, np.int64), bw[new])
        chk(lib.strata_op_dedup_diff(ctx, kb, p(kb_), nb, p(ka), na, p(do), C.byref(nd)))
        assert np.array_equal(got(do, nd.value, kt), b[~hit])
        chk(lib.strata_op_min_improve(ctx, kb, p(kb_), p(wb), nb, p(ka), p(wa), na, p(do), p(dw), C.byref(nd)))
        assert np.array_equal(got(do, nd.value, kt), b[better])
        assert np.array_equal(got(dw, nd.value, np.int64), bw[better])
        low = aw.copy()
        np.minimum.at(low, at[hit], bw[hit])
        assert np.array_equal(wa.cpu().numpy(), low)
