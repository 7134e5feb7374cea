"""The row-major kernel for few query rows (fmb_decode_fwd: gating and attention in one launch),
called through the C ABI whatever the size rule says, against the CPU oracle on the same centroids.

Tolerance: scores, probabilities and sums are fp32 and only the result is rounded to the I/O type,
so |x - fp32| <= half a unit in the last place: with p significant bits the unit of a value in
[2^e, 2^(e+1)) is 2^(e-p+1), so half of it is at most 2^-p of the value (p = 8 in bf16, 11 in fp16);
plus fp32 summation error over at most 64 * 320 keys of values below 6 (1e-4 absolute covers it)."""
import math
import os
import sys

import pytest
import torch

from conftest import cu_of

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
from oracle import moba_oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _decode(q, k, v, km, cu_km, cq, ck, mk, topk, chunk, causal):
    from flash_moba_b200 import _lib
    out = torch.empty_like(q)
    T, H, d = q.shape
    _lib.check(_lib.lib.fmb_decode_fwd(
        q.data_ptr(), q.stride(0), q.stride(1), k.data_ptr(), k.stride(0), k.stride(1), v.data_ptr(), v.stride(0), v.stride(1),
        km.data_ptr(), out.data_ptr(), out.stride(0), out.stride(1), cq.data_ptr(), ck.data_ptr(), cu_km.data_ptr(),
        cq.numel() - 1, H, k.shape[1], d, T, mk, topk, chunk, 1.0 / math.sqrt(d), int(causal),
        0 if q.dtype == torch.bfloat16 else 1, torch.cuda.current_stream().cuda_stream))
    return out


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("lens_q,lens_k,H,Hk,d,chunk,topk,dtype", [
    ([1], [1], 4, 2, 128, 64, 4, "bf16"),                                  # a single key
    ([1], [5000], 8, 2, 128, 128, 8, "bf16"),                              # one row: clusters of several CTAs
    ([1, 1, 1], [64, 65, 1279], 4, 4, 64, 64, 3, "fp16"),                  # chunk boundaries
    ([1] * 40, [300 + 37 * i for i in range(40)], 16, 2, 128, 128, 8, "bf16"),   # more rows than CTAs: no cluster
    ([3, 1, 0, 7], [700, 1, 50, 2000], 6, 2, 128, 64, 5, "fp16"),          # three heads per kv head, an empty block
    ([2, 4], [900, 2], 8, 1, 256, 256, 2, "bf16"),                         # more rows than keys; a warp per row of 256
    ([1, 2], [1500, 777], 12, 12, 96, 64, 16, "bf16"),                     # d between the tile widths
    ([1], [4321], 2, 1, 64, 64, 64, "bf16"),                               # the longest list, fewer chunks in reach than places
    ([5], [6000], 16, 1, 256, 64, 33, "fp16"),
    ([1] * 170, [129 + i for i in range(170)], 8, 1, 64, 64, 4, "fp16"),   # eight heads per kv head, many rows: clusters of one CTA
    ([1] * 80, [200 + i for i in range(80)], 32, 1, 128, 64, 2, "bf16"),
    ([1], [2000], 3, 3, 8, 320, 1, "bf16"),                                # one 16-byte chunk per row, own chunk only
])
def test_decode_kernel_vs_oracle(lens_q, lens_k, H, Hk, d, chunk, topk, dtype, causal):
    from flash_moba_b200 import ops
    g = torch.Generator().manual_seed(len(lens_q) * 1000 + d)
    dt = torch.bfloat16 if dtype == "bf16" else torch.float16
    q = torch.randn(sum(lens_q), H, d, generator=g).to(dt)
    k = torch.randn(sum(lens_k), Hk, d, generator=g).to(dt)
    v = torch.randn(sum(lens_k), Hk, d, generator=g).to(dt)
    cq, ck, mk = cu_of(lens_q), cu_of(lens_k), max(lens_k)
    km, cu_km = ops.mean_pool(k.to(DEV), ck.to(DEV), mk, chunk)
    got = _decode(q.to(DEV), k.to(DEV), v.to(DEV), km, cu_km, cq.to(DEV), ck.to(DEV), mk, topk, chunk, causal).cpu().float()
    n = int(cu_km[-1])
    idx, _ = O.gate_topk(q, km[:n].cpu(), cq, ck, cu_km.cpu(), topk, chunk, causal)
    want, _ = O.attention_blocked(q.float(), k.float(), v.float(), cq, ck, idx, chunk, causal)
    rel = 2.0 ** -8 if dtype == "bf16" else 2.0 ** -11
    assert ((got - want).abs() <= rel * want.abs() + 1e-4).all(), (got - want).abs().max()


def test_decode_kernel_ties_and_own_chunk():
    """Integer-valued queries against identical centroids: every score ties, so the list is the row's
    own chunk and the highest chunk ids; values name their chunk, and equal keys make the result the
    plain mean of the selected keys' values."""
    from flash_moba_b200 import ops
    H, Hk, d, chunk, topk, n = 4, 2, 64, 64, 3, 640
    q = torch.ones(1, H, d, dtype=torch.bfloat16)
    k = torch.ones(n, Hk, d, dtype=torch.bfloat16)
    v = (torch.arange(n) // chunk).float().view(n, 1, 1).expand(n, Hk, d).to(torch.bfloat16).contiguous()
    cq, ck = cu_of([1]), cu_of([n])
    km, cu_km = ops.mean_pool(k.to(DEV), ck.to(DEV), n, chunk)
    got = _decode(q.to(DEV), k.to(DEV), v.to(DEV), km, cu_km, cq.to(DEV), ck.to(DEV), n, topk, chunk, True).cpu().float()
    assert torch.equal(got, torch.full_like(got, (9 + 8 + 7) / 3))
