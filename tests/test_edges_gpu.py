"""Kernels at the sizes where their loops and rings can go wrong: rows of a chunk around the pool's turns of sixteen, eight and four,
rows of the dO.O kernel whose (token, head) is found by counting, forward items of a single tile that follow one another
through the K and V buffers, backward items of one and of seven tiles, tiles whose rows stand at the edge of the causal mask, equal scores in one lane's and in
several lanes' candidates of the decode kernel."""
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


@pytest.mark.parametrize("d", [64, 96, 128, 256])
@pytest.mark.parametrize("chunk", [64, 192])
def test_pool_row_counts(d, chunk):
    """|x - mean| <= half a bf16 unit of the mean (2^-8 of it) + fp32 sums of 192 values below 6 (1e-5)."""
    from flash_moba_b200 import ops
    lens = [1, 15, 16, 17, 31, 33, 63, 64, 65, 127, 129, 191, 193]
    k = torch.randn(sum(lens), 3, d, generator=torch.Generator().manual_seed(d)).bfloat16()
    km, cu_km = ops.mean_pool(k.to(DEV), cu_of(lens).to(DEV), max(lens), chunk)
    at, row = 0, 0
    for n in lens:
        for c in range(0, n, chunk):
            want = k[at + c:at + min(n, c + chunk)].double().mean(0)
            assert ((km[row].cpu().double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all(), (n, c)
            row += 1
        at += n
    assert int(cu_km[-1]) == row


@pytest.mark.parametrize("d", [8, 32, 64, 96, 256])
@pytest.mark.parametrize("chunk", [16, 64, 80, 320])
def test_pool_sums_in_row_order(d, chunk):
    """However many rows are requested at a time: a lane adds its rows (every 32 / lanes-per-row th) in their order in fp32, then the
    lanes' sums meet pairwise.  The same bits."""
    from flash_moba_b200 import ops
    lens = [1, 3, 15, 16, 17, 57, 61, 63, 64, 79, 81, 130, 255, 319, 321]
    k = torch.randn(sum(lens), 2, d, generator=torch.Generator().manual_seed(d)).bfloat16()
    km, _ = ops.mean_pool(k.to(DEV), cu_of(lens).to(DEV), max(lens), chunk)
    rpi = 32 // (1 << (d // 8 - 1).bit_length())
    at, row = 0, 0
    for n in lens:
        for c in range(0, n, chunk):
            x = k[at + c:at + min(n, c + chunk)].float()
            parts = [torch.zeros_like(x[0]) for _ in range(rpi)]
            for i in range(len(x)):
                parts[i % rpi] = parts[i % rpi] + x[i]
            while len(parts) > 1:
                parts = [a + b for a, b in zip(parts[::2], parts[1::2])]
            want = (parts[0] * (torch.ones(()) / len(x))).bfloat16()
            assert torch.equal(km[row].cpu(), want), (n, c)
            row += 1
        at += n


@pytest.mark.parametrize("H", [1, 2, 3, 7, 12])
@pytest.mark.parametrize("T,d", [(1, 64), (129, 64), (65, 128), (33, 256)])
def test_dot_of_gradient_and_output(T, H, d):
    """fp32 sums of d products: at most d roundings of 2^-24 of the sum of their magnitudes."""
    import flash_moba_b200 as F
    from flash_moba_b200 import _fmb_torch
    g = torch.Generator().manual_seed(T + H)
    q, k, v, do = (torch.randn(T, H, d, generator=g).bfloat16().to(DEV) for _ in range(4))
    cu = cu_of([T]).to(DEV)
    co, cn, ind = F.flash_topk_varlen_func(q, k, cu, cu, T, T, 2, 64, causal=True)
    geo = (cu, cu, T, T)
    out, lse, _ = _fmb_torch.attn_fwd(q, k, v, co, cn, ind, *geo, 64, 0.1, True, None, None, None)
    dq, dk, dv = (torch.empty_like(x) for x in (q, k, v))
    got = _fmb_torch.attn_bwd(do, q, k, v, out, lse, dq, dk, dv, co, cn, ind, *geo, 64, 0.1, True, None)
    x = do.double() * out.double()
    assert ((got.double().T - x.sum(-1)).abs() <= d * 2.0 ** -24 * x.abs().sum(-1) + 1e-30).all()


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("chunk", [64, 128])
@pytest.mark.parametrize("lens_q,lens_k,H,Hk,topk", [
    ([37, 1], [8000, 5000], 16, 16, 4),            # hundreds of items of one short tile
    ([130, 70], [4100, 3000], 32, 8, 5),           # several heads to an item
    ([129, 64, 300], [129, 64, 300], 8, 8, 3),     # rows at the mask's edges, tiles of one row
    ([700, 300], [30000, 11000], 16, 16, 8),       # up to 69 items of one tile per CTA, one after the other
])
def test_forward_of_short_items(lens_q, lens_k, H, Hk, topk, chunk, d):
    """Tolerance: inputs of 8 significant bits, probabilities and every chunk's part of a row rounded to them, at most 2^-8 each, of
    values below 6: 3 x 2^-8 x 6 = 0.07 bounds each element, and the 2-norm error of independent roundings (three of
    2^-9 on average) is below 4 x 2^-9.  The lists are the oracle's, so no selection can differ."""
    import flash_moba_b200 as F
    from flash_moba_b200 import ops
    g = torch.Generator().manual_seed(chunk + d)
    q, k, v = (torch.randn(n, h, d, generator=g).bfloat16() for n, h in ((sum(lens_q), H), (sum(lens_k), Hk), (sum(lens_k), Hk)))
    cq, ck, mq, mk = cu_of(lens_q), cu_of(lens_k), max(lens_q), max(lens_k)
    km, cu_km = ops.mean_pool(k.to(DEV), ck.to(DEV), mk, chunk)
    n_km = int(cu_km[-1])
    idx, _ = O.gate_topk(q, km[:n_km].cpu(), cq, ck, cu_km.cpu(), topk, chunk, True)
    want = O.attention_blocked(q.float(), k.float(), v.float(), cq, ck, idx, chunk, True)[0]
    co, cn, ind = ops.build_csc(idx.to(DEV), cq.to(DEV), mq, -(-mk // chunk))[:3]
    dev = [t.to(DEV) for t in (q, k, v, cq, ck)]
    runs = [F.flash_moba_attn_varlen_func(*dev[:3], *dev[3:], mq, mk, co, cn, ind, 128, chunk, causal=True) for _ in range(2)]
    assert torch.equal(runs[0], runs[1])
    diff = runs[0].cpu().float() - want
    assert diff.abs().max() <= 0.07
    assert diff.norm() <= 4 * 2.0 ** -9 * want.norm()


@pytest.mark.parametrize("chunk", [64, 128])
@pytest.mark.parametrize("tiles", [1, 7])
def test_backward_of_items_of_few_tiles(tiles, chunk):
    """Head dim 64, where the backward kernel has three Q buffers and three (64-key blocks) or two (128) dO buffers: items of one tile
    leave the ring of buffers turned by one for the next item, items of seven go around it more than twice.  Every row
    sees every chunk of its sequence.  Error bars: those of the other attention tests."""
    from test_kernels_gpu import _attn_check
    g = torch.Generator().manual_seed(chunk)
    H = 12 if tiles == 1 else 4
    lens = [1 + i % chunk for i in range(0, 120 * 7, 7)] if tiles == 1 else [7 * 128] * 16
    ncol = -(-max(lens) // chunk)
    q, k, v, do = (torch.randn(sum(lens), H, 64, generator=g).bfloat16() for _ in range(4))
    mask = torch.ones(len(lens), H, max(lens), ncol, dtype=torch.bool)
    for b, n in enumerate(lens):
        mask[b, :, n:] = False
        mask[b, :, :, -(-n // chunk):] = False
    _attn_check(q, k, v, do, cu_of(lens), cu_of(lens), mask, chunk, False, 1)


@pytest.mark.parametrize("n_chunks,topk", [(2, 8), (31, 4), (33, 8), (64, 8), (65, 5), (100, 16), (200, 33)])
def test_decode_selection_of_equal_scores(n_chunks, topk):
    """Keys alike inside a chunk and of a few values only: the centroids are exact, most scores tie (at zero among others; all zeros are +0,
    as the pool and the products start their sums from it), and any other choice of chunks gives another result.  Tolerance as for the decode kernel: half a unit of the
    result's type (2^-8 of it) + fp32 sums."""
    from flash_moba_b200 import ops
    from test_decode_gpu import _decode
    H, Hk, d, chunk = 8, 4, 64, 64
    g = torch.Generator().manual_seed(n_chunks)
    n = n_chunks * chunk - 5
    q = torch.randint(-1, 2, (2, H, d), generator=g).bfloat16() * 0.5
    few = torch.randint(-1, 2, (3, Hk, d), generator=g).bfloat16()
    few[0] = -0.0                                     # a third of the chunks scores zero
    k = few[torch.randint(0, 3, (n_chunks,), generator=g)].repeat_interleave(chunk, 0)[:n].contiguous()
    v = torch.randn(n, Hk, d, generator=g).bfloat16()
    cq, ck = cu_of([2]), cu_of([n])
    km, cu_km = ops.mean_pool(k.to(DEV), ck.to(DEV), n, chunk)
    got = _decode(q.to(DEV), k.to(DEV), v.to(DEV), km, cu_km, cq.to(DEV), ck.to(DEV), n, topk, chunk, True).cpu().float()
    idx, _ = O.gate_topk(q, km[:int(cu_km[-1])].cpu(), cq, ck, cu_km.cpu(), topk, chunk, True)
    want, _ = O.attention_blocked(q.float(), k.float(), v.float(), cq, ck, idx, chunk, True)
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4).all(), (got - want).abs().max()
