"""Operators over buffers that share memory or lie off their type's alignment:
a sort from columns at odd byte addresses, a join whose output keys lie over an
input weight column."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kb,vb", [(4, 0), (4, 4), (8, 4), (8, 8)])
@pytest.mark.parametrize("shift", [1, 2, 4])
@pytest.mark.parametrize("n", [1, 5000])
def test_sort_from_unaligned_columns(engine, kb, vb, shift, n):
    import torch
    rng = np.random.default_rng(n + shift)
    k = rng.integers(0, 2 ** (8 * kb), n, dtype=np.uint64).astype({4: np.uint32, 8: np.uint64}[kb])
    v = np.arange(n).astype({4: np.uint32, 8: np.uint64}[vb or 4])

    def odd(a):  # the column `shift` bytes into a buffer
        t = torch.zeros(a.nbytes + 16, dtype=torch.uint8, device="cuda")
        t[shift:shift + a.nbytes] = torch.from_numpy(a.view(np.uint8)).cuda()
        return t
    ki, vi = odd(k), odd(v)
    ko = torch.empty(n * kb, dtype=torch.uint8, device="cuda")
    vo = torch.empty(n * max(vb, 1), dtype=torch.uint8, device="cuda")
    engine._check(engine.lib.strata_op_sort(engine.ctx, kb, vb, ki.data_ptr() + shift, vi.data_ptr() + shift if vb else None,
                                            ko.data_ptr(), vo.data_ptr() if vb else None, n, 8 * kb))
    o = np.argsort(k, kind="stable")
    assert np.array_equal(ko.cpu().numpy().view(k.dtype), k[o])
    if vb:
        assert np.array_equal(vo.cpu().numpy().view(v.dtype), v[o])


@pytest.mark.parametrize("over", ["a", "b"])
@pytest.mark.parametrize("n", [3, 1536, 20_000])
def test_join_keys_over_weights(engine, over, n):
    import torch
    y = np.arange(n, dtype=np.int64)
    aw, bw = torch.from_numpy(y * 3 - 7).cuda(), torch.from_numpy(11 - y).cuda()
    a = torch.from_numpy((y[::-1].copy() << 32) | y).cuda()  # (n - 1 - y, y)
    b = torch.from_numpy((y << 32) | 5).cuda()
    out, ow = {"a": aw, "b": bw}[over], torch.empty(n, dtype=torch.int64, device="cuda")
    c = C.c_uint64()
    engine._check(engine.lib.strata_op_join(engine.ctx, 8, a.data_ptr(), aw.data_ptr(), n, 32, b.data_ptr(),
                                            bw.data_ptr(), n, 32, 32, out.data_ptr(), ow.data_ptr(), n, C.byref(c)))
    assert c.value == n
    assert out.tolist() == ((y[::-1] << 32) | 5).tolist()
    assert ow.tolist() == (y * 2 + 4).tolist()
