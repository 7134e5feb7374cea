"""Batches of many short sequences: a CTA of the attention kernels has eight or more items of a tile or two, most of short blocks of keys, which
follow one another through every buffer and ring several times.  Error bars: those of the other attention tests."""
import pytest
import torch

from conftest import cu_of
from oracle import moba_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _batch(H, Hk, d, chunk):
    """Sequences of two chunks, the second of them short.  In every third all rows of the second chunk look at the first one only (keys
    that no row of any head selects), in every other third half of the heads do (groups of which some heads have no entries)."""
    g = torch.Generator().manual_seed(chunk + d + H)
    lens = [chunk + 1 + (i * 5) % (3 * chunk // 4) for i in range(600 // Hk)]
    T, m = sum(lens), max(lens)
    q, k, v, do = (torch.randn(T, h, d, generator=g).bfloat16() for h in (H, Hk, Hk, H))
    mask = torch.zeros(len(lens), H, m, 2, dtype=torch.bool)
    mask[:, :, :chunk, 0] = True
    mask[:, :, chunk:] = torch.tensor([False, True])
    mask[:, :, chunk:, 0] = torch.rand(len(lens), H, m - chunk, generator=g) < 0.5
    for i, heads in ((0, slice(None)), (1, slice(None, None, 2))):
        mask[i::3, heads, chunk:] = torch.tensor([True, False])
    for b, n in enumerate(lens):
        mask[b, :, n:] = False
    return lens, cu_of(lens), q, k, v, do, mask


@pytest.mark.parametrize("H,Hk", [(8, 8), (16, 4)])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("chunk", [64, 128])
def test_many_short_sequences_forward(chunk, d, H, Hk):
    import flash_moba_b200 as F
    from test_kernels_gpu import _attn_check
    lens, cu, q, k, v, do, mask = _batch(H, Hk, d, chunk)
    _attn_check(q, k, v, do, cu, cu, mask, chunk, True, 1, check_grad=False)
    pattern = [t.to(DEV) for t in O.mask_to_csc(mask, cu, cu, chunk)[:3]]
    dev = [t.to(DEV) for t in (q, k, v)]
    runs = [F.flash_moba_attn_varlen_func(*dev, cu.to(DEV), cu.to(DEV), max(lens), max(lens), *pattern, 128, chunk, causal=True) for _ in range(3)]
    assert torch.equal(runs[0], runs[1]) and torch.equal(runs[0], runs[2])


@pytest.mark.parametrize("H,Hk", [(8, 8), (16, 4)])
@pytest.mark.parametrize("d", [64, 128, 256])
@pytest.mark.parametrize("chunk", [64, 128])
def test_many_short_sequences_backward(chunk, d, H, Hk):
    """Keys that no row selects have gradients of exactly zero, and two runs agree to the bit."""
    from flash_moba_b200 import ops
    from test_kernels_gpu import _attn_check
    lens, cu, q, k, v, do, mask = _batch(H, Hk, d, chunk)
    _attn_check(q, k, v, do, cu, cu, mask, chunk, True, 1)
    pattern = [t.to(DEV) for t in O.mask_to_csc(mask, cu, cu, chunk)[:3]]
    dev = [t.to(DEV) for t in (q, k, v, do, cu)]
    geo = (*pattern, dev[4], dev[4], max(lens), max(lens), chunk, d ** -0.5, True)
    out, lse = ops.attn_fwd(*dev[:3], *geo)
    runs = []
    for _ in range(2):
        grads = [torch.full_like(t, 7.0) for t in dev[:3]]
        ops.attn_bwd(dev[3], *dev[:3], out, lse, *grads, *geo)
        runs.append(grads)
    assert all(torch.equal(a, b) for a, b in zip(*runs))
    for i in range(0, len(lens), 3):
        rows = slice(int(cu[i]) + chunk, int(cu[i + 1]))
        assert not runs[0][1][rows].any() and not runs[0][2][rows].any()
