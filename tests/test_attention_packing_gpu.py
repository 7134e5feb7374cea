"""Forward work items that hold the columns of several q heads of a kv head (up to 8, a divisor of the group), tiles
whose rows belong to two or more heads, several items per claim (short columns, most of them empty), and more
tiles per CTA than it has tile buffers: against the dense oracle, forward and backward, with the bars of
tests/test_kernels_gpu.py."""
import pytest
import torch

from conftest import cu_of
from test_kernels_gpu import _attn_check, _random_mask

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,Hk,d,chunk,lens,causal,topk", [
    (7, 1, 128, 128, [300], True, 2),
    (11, 1, 64, 128, [260], True, 2),             # a prime group above eight: items of one head
    (8, 2, 128, 128, [1, 127, 129, 900, 3], True, 2),   # ragged: many empty columns
    (6, 2, 128, 256, [700, 90], True, 2),         # two key blocks per chunk
    (4, 4, 64, 64, [2000], False, 3),
    # enough columns (8 per SM) for items of several heads: 7, 6 (of 12), 8 (of 16) and 4 heads
    (14, 2, 64, 64, [63] * 160 + [200] * 5, True, 2),
    (24, 2, 64, 64, [65, 1] * 80, True, 2),
    (32, 2, 128, 64, [66, 3] * 75, False, 2),
    (16, 4, 128, 128, [130, 5] * 75, True, 2),
])
def test_packed_columns(H, Hk, d, chunk, lens, causal, topk):
    torch.manual_seed(H * 100 + d)
    T = sum(lens)
    q, do = torch.randn(T, H, d).bfloat16(), torch.randn(T, H, d).bfloat16()
    k, v = torch.randn(T, Hk, d).bfloat16(), torch.randn(T, Hk, d).bfloat16()
    mask = _random_mask(lens, lens, H, chunk, causal, topk)
    _attn_check(q, k, v, do, cu_of(lens), cu_of(lens), mask, chunk, causal, 1)


def test_wrong_number_of_columns_raises():
    import flash_moba_b200 as F
    q = torch.randn(256, 2, 64, device="cuda").bfloat16()
    cu = cu_of([256]).cuda()
    pattern = F.flash_topk_varlen_func(q, q, cu, cu, 256, 256, 2, 64, causal=True)
    with pytest.raises(RuntimeError, match="pattern has 4 columns, expected .* = 2"):
        F.flash_moba_attn_varlen_func(q, q, q, cu, cu, 256, 256, *pattern, 128, 128, causal=True)
