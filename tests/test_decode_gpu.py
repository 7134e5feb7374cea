"""The row-major kernel for few query rows (fmb_decode_fwd: gating and attention in one launch),
called through the C ABI whatever the size rule says, against the CPU oracle on the same centroids.

Tolerance: scores and sums are fp32, probabilities keep at least 16 bits, and only the result is rounded to the I/O type,
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
    ([1], [5000], 8, 2, 128, 128, 8, "bf16"),                              # one row: clusters of four CTAs
    ([1], [9000], 8, 8, 128, 256, 8, "bf16"),                              # of eight: 64 groups of keys for a head
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


def _special(name, q, k, v, own0):
    """Plants special numbers in keys and values of each row's own chunk (key `own0` on), or in a query."""
    if name == "nan_q":
        q[0, 1, 5] = float("nan")
    elif name == "nan_k":
        k[own0 + 3, 0, 7] = float("nan")
    elif name == "nan_v":
        v[own0 + 3, 0, 7] = float("nan")
    elif name == "inf_v":
        v[own0 + 3, 0, 7] = float("inf")
        v[own0 + 5, 1, 9] = float("-inf")
    elif name == "inf_k":
        k[own0 + 3, 0, 7] = float("inf")
    elif name == "low_k":                          # scores that overflow to -inf for a run of whole groups of keys
        big = torch.finfo(k.dtype).max
        for h in range(q.shape[1]):
            k[own0:own0 + 64, h // (q.shape[1] // k.shape[1])] = -big
        q.abs_()


@pytest.mark.parametrize("d", [64, 128, 256])
@pytest.mark.parametrize("dtype", ["bf16", "fp16"])
@pytest.mark.parametrize("name", ["nan_q", "nan_k", "nan_v", "inf_v", "inf_k", "low_k"])
def test_decode_kernel_special_numbers(name, dtype, d):
    """NaN and infinities go through as softmax(scores) . V gives them: a row that meets a NaN is NaN, an infinite value with a
    weight above zero makes its column infinite, keys whose scores are -inf have no weight."""
    if name == "low_k" and dtype == "fp16":
        pytest.skip("products of fp16 numbers do not leave the range of fp32")
    from flash_moba_b200 import ops
    g = torch.Generator().manual_seed(d)
    dt = torch.bfloat16 if dtype == "bf16" else torch.float16
    H, Hk, chunk, topk, n = 4, 2, 128, 3, 1000
    q, k, v = (torch.randn(m, h, d, generator=g) for m, h in ((1, H), (n, Hk), (n, Hk)))
    if name == "low_k":
        q *= 100.0
    q, k, v = (t.to(dt) for t in (q, k, v))
    cq, ck = cu_of([1]), cu_of([n])
    km, cu_km = ops.mean_pool(k.to(DEV), ck.to(DEV), n, chunk)        # centroids before the planted numbers: known lists
    own0 = (n - 1) // chunk * chunk
    _special(name, q, k, v, own0)
    got = _decode(q.to(DEV), k.to(DEV), v.to(DEV), km, cu_km, cq.to(DEV), ck.to(DEV), n, topk, chunk, True).cpu().double()
    n_km = int(cu_km[-1])
    idx, _ = O.gate_topk(q.nan_to_num(), km[:n_km].cpu(), cq, ck, cu_km.cpu(), topk, chunk, True)
    for h in range(H):
        chunks = [own0 // chunk] if name == "nan_q" and h == 1 else [int(c) for c in idx[0, h] if c >= 0]   # (NaN scores select nothing)
        keys = torch.cat([torch.arange(c * chunk, min(n, (c + 1) * chunk)) for c in sorted(chunks)])
        s = (k[keys, h // 2].float() @ q[0, h].float()).double() / math.sqrt(d)
        p = torch.softmax(s, 0)
        x = v[keys, h // 2].double()
        want = torch.where(p.unsqueeze(1) > 0, p.unsqueeze(1) * x, p.unsqueeze(1) * torch.nan_to_num(x, posinf=0, neginf=0)).sum(0)
        a = got[0, h]
        assert torch.equal(torch.isnan(a), torch.isnan(want)), h
        assert torch.equal(torch.isinf(a), torch.isinf(want)) and torch.equal(a[torch.isinf(a)], want[torch.isinf(want)]), h
        ok = torch.isfinite(want)
        rel = 2.0 ** -8 if dtype == "bf16" else 2.0 ** -11
        # (low_k: scores some 100 times larger, and so is the rounding of their fp32 sums: 100 x 2^-24 x sqrt(d) of the weights)
        assert ((a - want).abs()[ok] <= rel * want.abs()[ok] + (2e-3 if name == "low_k" else 1e-4)).all(), h
