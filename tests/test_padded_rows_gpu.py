"""Rows of q behind the last sequence (a token buffer padded to a fixed size): no sequence owns them, so they see no key.
They get zeros, whichever way a call takes, and the rows of the sequences get what they get without the padding."""
import math

import pytest
import torch

from conftest import cu_of

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("lens_q,H,Hk,d,pad", [([1, 2], 8, 2, 128, 1), ([3], 4, 4, 64, 5), ([1] * 40, 16, 2, 128, 3), ([2], 2, 1, 256, 2)])
def test_decode_kernel_writes_zeros(lens_q, H, Hk, d, pad):
    from flash_moba_b200 import _lib, ops
    torch.manual_seed(d)
    lens_k, n, chunk, topk = [200 + 30 * i for i in range(len(lens_q))], sum(lens_q), 64, 3
    q = torch.randn(n + pad, H, d, device=DEV).bfloat16()
    k, v = (torch.randn(sum(lens_k), Hk, d, device=DEV).bfloat16() for _ in range(2))
    cq, ck = cu_of(lens_q).to(DEV), cu_of(lens_k).to(DEV)
    km, cu_km = ops.mean_pool(k, ck, max(lens_k), chunk)

    def decode(q):
        out = torch.full_like(q, float("nan"))
        _lib.check(_lib.lib.fmb_decode_fwd(
            q.data_ptr(), q.stride(0), q.stride(1), k.data_ptr(), k.stride(0), k.stride(1), v.data_ptr(), v.stride(0), v.stride(1),
            km.data_ptr(), out.data_ptr(), out.stride(0), out.stride(1), cq.data_ptr(), ck.data_ptr(), cu_km.data_ptr(),
            len(lens_q), H, Hk, d, q.shape[0], max(lens_k), topk, chunk, 1.0 / math.sqrt(d), 1, 0,
            torch.cuda.current_stream().cuda_stream))
        return out

    got = decode(q)
    assert torch.equal(got[n:], torch.zeros_like(got[n:]))
    # (the split of a row's keys over CTAs goes by the number of rows: fp32 sums in another order, then one rounding)
    torch.testing.assert_close(got[:n].float(), decode(q[:n]).float(), rtol=2 ** -7, atol=1e-4)


@pytest.mark.parametrize("lens,topk,pad,lead", [([512, 100], 4, 700, 0), ([300], 8, 1, 0), ([40, 0], 16, 600, 0), ([100, 60], 20, 30, 0),
                                                ([50, 0, 9], 3, 5, 7)])
def test_row_lists_of_such_rows_are_empty(lens, topk, pad, lead):
    from flash_moba_b200 import _lib
    H, ncol, n = 2, 11, sum(lens)
    T, mx = lead + n + pad, max(lens)
    cu = (cu_of(lens) + lead).to(torch.int32).to(DEV)
    lists = torch.randint(0, ncol, (H, T, topk), dtype=torch.int32, device=DEV)
    co = torch.empty(len(lens), H, ncol, dtype=torch.int64, device=DEV)
    cn = torch.empty(len(lens), H, ncol, dtype=torch.int32, device=DEV)
    ind = torch.zeros(T * H * topk, dtype=torch.int32, device=DEV)
    rows = torch.full((H, T, topk), 12345, dtype=torch.int32, device=DEV)
    nbytes = _lib.lib.fmb_build_csc_workspace_bytes(len(lens), H, mx, ncol)
    ws = torch.empty(nbytes, dtype=torch.uint8, device=DEV)
    _lib.check(_lib.lib.fmb_build_csc_rows(lists.data_ptr(), topk, T * topk, cu.data_ptr(), co.data_ptr(), cn.data_ptr(),
                                           ind.data_ptr(), rows.data_ptr(), ws.data_ptr(), nbytes, len(lens), H, topk, T, mx, ncol,
                                           torch.cuda.current_stream().cuda_stream))
    outside = torch.cat([rows[:, :lead], rows[:, lead + n:]], dim=1)
    assert torch.equal(outside, torch.full_like(outside, -1))


@pytest.mark.parametrize("d,chunk,share", [(64, 64, True), (128, 128, True), (256, 128, True), (128, 128, False)])
def test_training_step(d, chunk, share, monkeypatch):
    import flash_moba_b200 as F
    monkeypatch.setenv("FMB_SHARE_LISTS", "1" if share else "0")      # 0: the attention calls build their own lists
    torch.manual_seed(chunk + d)
    lens, H, Hk, topk, pad = [700, 130], 4, 2, 3, 333
    n, cu = sum(lens), cu_of(lens).to(DEV)

    def step(q, k, v, do):
        q, k, v = (t.clone().requires_grad_(True) for t in (q, k, v))
        out = F.flash_moba_varlen_func(q, k, v, cu, cu, max(lens), max(lens), chunk, topk)
        return [out.detach(), *torch.autograd.grad(out, (q, k, v), do)]

    q, do = (torch.randn(n + pad, H, d, device=DEV).bfloat16() for _ in range(2))
    k, v = (torch.randn(n, Hk, d, device=DEV).bfloat16() for _ in range(2))
    want, got = step(q[:n], k, v, do[:n]), step(q, k, v, do)
    for i, (a, b) in enumerate(zip(want, got)):
        assert torch.equal(a, b[:n]), i
        assert torch.equal(b[n:], torch.zeros_like(b[n:])), i
