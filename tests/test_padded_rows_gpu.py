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
