"""Head dim 256 on the tensor cores: columns that end at, before and after a tile of 128 rows, columns of one row, key
blocks of 64 and 128 keys with a short last one, chunks of several key blocks, empty columns, several
heads per work item and one: against the dense oracle, forward and backward, with the bars of tests/test_kernels_gpu.py."""
import pytest
import torch

from conftest import cu_of
from test_kernels_gpu import _attn_check, _random_mask

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,Hk,chunk,lens,causal,topk", [
    (1, 1, 64, [1], True, 1),
    (2, 1, 64, [127, 128, 129, 65], False, 2),
    (4, 2, 128, [128, 257, 1, 130], True, 2),
    (3, 3, 128, [700], False, 3),                 # five tiles and more per column: every buffer and phase in turn
    (6, 2, 192, [500, 90], True, 2),              # three key blocks per chunk
    (2, 2, 256, [700, 300], True, 2),             # two key blocks of 128 (forward), four of 64 (backward) per chunk
    # enough columns (8 per SM) for forward items of several heads: 7, 4 (of 8) heads
    (14, 2, 64, [63] * 160 + [130] * 5, True, 2),
    (16, 2, 128, [130, 5] * 160, True, 2),
])
def test_wide_heads(H, Hk, chunk, lens, causal, topk):
    torch.manual_seed(H * 100 + chunk)
    T = sum(lens)
    q, do = torch.randn(T, H, 256).bfloat16(), torch.randn(T, H, 256).bfloat16()
    k, v = torch.randn(T, Hk, 256).bfloat16(), torch.randn(T, Hk, 256).bfloat16()
    mask = _random_mask(lens, lens, H, chunk, causal, topk)
    _attn_check(q, k, v, do, cu_of(lens), cu_of(lens), mask, chunk, causal, 1)
