"""Work items that overlap, and rules that go by their sizes: backward items that follow one another through the K and V buffers,
among them items without any tile and short last blocks, gradients of keys whose rows begin on multiples of 16 but not of 32 bytes;
forward items of ragged batches taken several at a time; decode candidates around what a warp holds in registers."""
import pytest
import torch

import test_edges_gpu as edges
from conftest import cu_of
from oracle import moba_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("d", [64, 128, 256])
@pytest.mark.parametrize("chunk", [64, 128, 256])
@pytest.mark.parametrize("causal", [True, False])
def test_backward_items_without_tiles_and_narrow_alignment(chunk, d, causal):
    """Error bars: those of the other attention tests.  Keys that no row selects have gradients of exactly zero, and where dK and dV
    lie makes no difference to any bit."""
    from flash_moba_b200 import ops
    from test_kernels_gpu import _attn_check
    g = torch.Generator().manual_seed(chunk + d)
    H, lens = 24, [9 * chunk // 2 + 3, 2 * chunk + 33, 5]      # several items per CTA; sequences end inside a block
    T, m, ncol = sum(lens), max(lens), -(-max(lens) // chunk)
    q, k, v, do = (torch.randn(T, H, d, generator=g).bfloat16() for _ in range(4))
    mask = torch.rand(len(lens), H, m, ncol, generator=g) < 0.6
    own = torch.arange(m) // chunk
    for b, n in enumerate(lens):
        mask[b, :, torch.arange(m), own] = True
        if n > 2 * chunk:
            mask[b, ::2, :, 1] = False                         # in every second head nobody sees chunk 1 ...
            mask[b, ::2, chunk:2 * chunk, 0] = True            # ... but every row sees something
        if causal:
            mask[b] &= torch.arange(ncol) <= own[:, None]
        mask[b, :, n:] = False
        mask[b, :, :, -(-n // chunk):] = False
    cu = cu_of(lens)
    _attn_check(q, k, v, do, cu, cu, mask, chunk, causal, 1)

    co, cn, ind = (t.to(DEV) for t in O.mask_to_csc(mask, cu, cu, chunk)[:3])
    dev = [t.to(DEV) for t in (q, k, v, do, cu)]
    geo = (co, cn, ind, dev[4], dev[4], m, m, chunk, d ** -0.5, causal)
    out, lse = ops.attn_fwd(dev[0], dev[1], dev[2], *geo)

    def grads(pad):
        dq = torch.empty_like(dev[0])
        dk, dv = (torch.full((T, H, d + pad), 7.0, dtype=torch.bfloat16, device=DEV).flatten()[pad:pad + T * H * (d + pad) - pad]
                  .as_strided((T, H, d), (H * (d + pad), d + pad, 1)) for _ in range(2))
        ops.attn_bwd(dev[3], dev[0], dev[1], dev[2], out, lse, dq, dk, dv, *geo)
        return dq, dk, dv

    for a, b in zip(grads(0), grads(8)):                       # 8 elements are 16 bytes
        assert torch.equal(a, b)
    _, dk, dv = grads(0)
    assert not dk[chunk:2 * chunk, ::2].any() and not dv[chunk:2 * chunk, ::2].any()


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("chunk", [64, 128])
def test_forward_items_of_ragged_batches(chunk, d):
    """Half of the items lie past their sequence's end, the others have some two hundred entries."""
    edges.test_forward_of_short_items([300, 200, 20, 256], [2560, 1152, 4096, 512], 32, 8, 8, chunk, d)


@pytest.mark.parametrize("n_chunks,topk", [(512, 8), (513, 16), (514, 8), (700, 33)])
def test_decode_selection_around_the_held_candidates(n_chunks, topk):
    """Rows of n_chunks chunks have n_chunks - 1 candidates; 512 are held in registers."""
    edges.test_decode_selection_of_equal_scores(n_chunks, topk)


@pytest.mark.parametrize("n_chunks,topk", [(128, 8), (129, 16), (130, 8), (257, 33)])
def test_decode_selection_around_few_candidates(n_chunks, topk):
    """Up to 128 candidates a list are held four a lane, more sixteen a lane."""
    edges.test_decode_selection_of_equal_scores(n_chunks, topk)
