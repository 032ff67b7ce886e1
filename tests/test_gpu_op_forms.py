"""Operators at the edges of their tiles and digits: sorts over the bits that
vary (two windows, none, odd and even pass counts, buffers that coincide),
merges whose equal pairs meet tile and thread boundaries, joins with +inf,
weights without a code and an output column over an input one."""
import ctypes as C

import numpy as np
import pytest

import strata_b200 as S

pytestmark = pytest.mark.gpu

INF = 2**63 - 1


def _t(a):
    import torch
    a = np.ascontiguousarray(a)
    return torch.from_numpy(a.view({4: np.int32, 8: np.int64}[a.dtype.itemsize])).cuda()


def _sort(eng, k, v, bits, in_place=False):
    kb, vb = k.dtype.itemsize, 0 if v is None else v.dtype.itemsize
    ki, vi = _t(k), None if v is None else _t(v)
    ko, vo = (ki, vi) if in_place else (_t(np.zeros_like(k)), None if v is None else _t(np.zeros_like(v)))
    p = lambda t: None if t is None else t.data_ptr()
    eng._check(eng.lib.strata_op_sort(eng.ctx, kb, vb, p(ki), p(vi), p(ko), p(vo), len(k), bits))
    if not in_place:
        assert np.array_equal(ki.cpu().numpy().view(k.dtype), k)  # the inputs stay
    return ko.cpu().numpy().view(k.dtype), None if v is None else vo.cpu().numpy().view(v.dtype)


MASKS = [0, 1, 1 << 63, 0xFF, 0x1FF, (0x7FFFF << 32) | 0x7FFFF, (0xFFF << 32) | 0xFFF, (0x1F << 32) | 0x1F,
         0x8000000080000001, (1 << 64) - 1, 0x0F0F0F0F0F0F0F0F, (0xFFFFFFFF << 32)]


@pytest.mark.parametrize("mask", MASKS)
@pytest.mark.parametrize("n", [1, 2, 2303, 2304, 2305, 70_001])
def test_sort_over_varying_bits(engine, mask, n):
    rng = np.random.default_rng(n)
    k = (rng.integers(0, 2**64, n, dtype=np.uint64) & np.uint64(mask)) | np.uint64(0x40 & ~mask)
    v = np.arange(n, dtype=np.uint64)
    for bits, vals, same in ((64, v, False), (64, None, False), (64, v, True), (37, v, False)):
        key = k if bits == 64 else k & np.uint64((1 << bits) - 1)
        o = np.argsort(key, kind="stable")
        got_k, got_v = _sort(engine, k, vals, bits, same)
        assert np.array_equal(got_k, k[o])
        assert vals is None or np.array_equal(got_v, v[o])
    k4 = (k >> np.uint64(16)).astype(np.uint32)
    o = np.argsort(k4, kind="stable")
    got_k, got_v = _sort(engine, k4, v.astype(np.uint32), 32)
    assert np.array_equal(got_k, k4[o]) and np.array_equal(got_v, o.astype(np.uint32))


@pytest.mark.parametrize("na,nb", [(0, 1), (1, 0), (1, 1), (767, 768), (768, 768), (769, 768), (1535, 1), (1536, 1536),
                                   (1537, 3), (5000, 4999), (40_000, 7), (3, 40_000)])
@pytest.mark.parametrize("trop", [False, True])
def test_merge_diff_boundaries(engine, na, nb, trop):
    import torch
    rng = np.random.default_rng(na * 7 + nb)
    for spread in (1, 3):  # mostly equal pairs, then few
        a = np.sort(rng.choice(np.arange(max(na, nb, 1) * spread + 1, dtype=np.uint64), na, replace=False))
        b = np.sort(rng.choice(np.arange(max(na, nb, 1) * spread + 1, dtype=np.uint64), nb, replace=False))
        aw, bw = rng.integers(0, 5, na), rng.integers(0, 5, nb)
        aw[rng.random(na) < 0.1] = INF
        bw[rng.random(nb) < 0.1] = INF
        d = dict(zip(a.tolist(), aw.tolist()))
        delta = {}
        for k, w in zip(b.tolist(), bw.tolist()):
            if k not in d or (trop and w < d[k]):
                delta[k] = w
                d[k] = w
        ka, kb, wa, wb = _t(a), _t(b), _t(aw), _t(bw)
        fo, do = torch.empty(na + nb, dtype=torch.int64, device="cuda"), torch.empty(nb + 1, dtype=torch.int64, device="cuda")
        fw, dw = torch.empty_like(fo), torch.empty_like(do)
        nf, nd = C.c_uint64(), C.c_uint64()
        p = lambda t: t.data_ptr() or do.data_ptr()  # an empty tensor's pointer is NULL, which means "no weights"
        w4 = (p(wa), p(wb), p(fw), p(dw)) if trop else (None, None, None, None)
        engine._check(engine.lib.strata_op_merge_diff(engine.ctx, 8, p(ka), w4[0], na, p(kb), w4[1], nb, p(fo), w4[2],
                                                      p(do), w4[3], C.byref(nf), C.byref(nd)))
        keys = sorted(d)
        assert fo[:nf.value].tolist() == keys and do[:nd.value].tolist() == sorted(delta)
        if trop:
            assert fw[:nf.value].tolist() == [d[k] for k in keys]
            assert dw[:nd.value].tolist() == [delta[k] for k in sorted(delta)]


def _join(eng, a, aw, b, bw, over=None):
    import torch
    p = lambda t: None if t is None else t.data_ptr()
    ka, kb, wa, wb = _t(a), _t(b), _t(aw), _t(bw)
    n = C.c_uint64()
    args = (eng.ctx, 8, p(ka), p(wa), len(a), 32, p(kb), p(wb), len(b), 32, 32)
    eng._check(eng.lib.strata_op_join(*args, None, None, 0, C.byref(n)))
    out = torch.empty(n.value + 1, dtype=torch.int64, device="cuda")
    ow = {None: torch.empty_like(out), "a": wa, "b": wb}[over]
    eng._check(eng.lib.strata_op_join(*args, p(out), p(ow), n.value, C.byref(n)))
    return out[:n.value].tolist(), ow[:n.value].tolist()


@pytest.mark.parametrize("over", [None, "a", "b"])
@pytest.mark.parametrize("na", [1, 31, 1535, 1536, 1537, 6000])
def test_join_weights(engine, na, over):
    rng = np.random.default_rng(na)
    y = rng.integers(0, 900, na).astype(np.uint64)
    a = (np.arange(na, dtype=np.uint64) << np.uint64(32)) | y
    b = (np.arange(0, 1000, 2, dtype=np.uint64) << np.uint64(32)) | np.uint64(3)  # one row per even y: at most na rows out
    aw, bw = rng.integers(-50, 50, na), rng.integers(-50, 50, len(b))
    aw[rng.random(na) < 0.1] = INF
    bw[rng.random(len(b)) < 0.1] = INF
    hit = y % 2 == 0
    if over == "b" and hit.sum() > len(b):
        pytest.skip("more rows out than the column it would overwrite")
    k, w = _join(engine, a, aw, b, bw, over)
    assert k == (((a[hit] >> np.uint64(32)) << np.uint64(32)) | np.uint64(3)).tolist()
    assert w == [INF if x == INF or z == INF else int(x + z) for x, z in zip(aw[hit], bw[(y[hit] // 2).astype(int)])]


@pytest.mark.parametrize("side", ["a", "b"])
def test_join_refuses_weights_without_a_code(engine, side):
    a, b = np.array([1, 7], np.uint64), np.array([1 << 32, 2 << 32], np.uint64)  # only a's y = 1 joins
    aw, bw = np.array([1, 1]), np.array([1, 1])
    (aw if side == "a" else bw)[1] = INF - 1  # on a row that joins nothing
    with pytest.raises(S.WeightRange):
        _join(engine, a, aw, b, bw)
