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


@pytest.mark.parametrize("shift", [16, 48])
def test_workspace_on_a_16_byte_boundary(shift):
    """The C entry points take a workspace that starts on any 16-byte boundary."""
    import flash_moba_b200 as F
    from flash_moba_b200 import _lib
    lib, lens, H, Hk, d, chunk = _lib.lib, [300, 131], 4, 2, 256, 128
    T, mx, n_indices = sum(lens), max(lens), sum(lens) * H * 2
    torch.manual_seed(3)
    q, do = (torch.randn(T, H, d, device="cuda").bfloat16().requires_grad_(True) for _ in range(2))
    k, v = (torch.randn(T, Hk, d, device="cuda").bfloat16().requires_grad_(True) for _ in range(2))
    cu = cu_of(lens).cuda()
    pattern = tuple(t.clone() for t in F.flash_topk_varlen_func(q, k, cu, cu, mx, mx, 2, chunk, causal=True))
    want = F.flash_moba_attn_varlen_func(q, k, v, cu, cu, mx, mx, *pattern, 128, chunk, causal=True)
    want_grads = torch.autograd.grad(want, (q, k, v), do)
    geo = (T, H, Hk, d, n_indices, len(lens), mx, chunk, H)
    stream, p = torch.cuda.current_stream().cuda_stream, lambda t: (t.data_ptr(), t.stride(0), t.stride(1))  # noqa: E731
    co, cn, ind = (t.data_ptr() for t in pattern)
    out, lse = torch.empty_like(q), torch.empty(H, T, device="cuda")
    nbytes = lib.fmb_attn_fwd_workspace_bytes(*geo)
    ws = torch.empty(nbytes + 64, dtype=torch.uint8, device="cuda")
    tail = (len(lens), H, Hk, d, T)
    _lib.check(lib.fmb_attn_fwd(*p(q), *p(k), *p(v), *p(out), lse.data_ptr(), co, cn, ind, n_indices, cu.data_ptr(), cu.data_ptr(),
                                ws.data_ptr() + shift, nbytes, *tail, mx, mx, chunk, d ** -0.5, 1, 0, stream))
    assert torch.equal(out, want)
    dq, dk, dv, sd = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v), torch.empty_like(lse)
    nbytes = lib.fmb_attn_bwd_workspace_bytes(*geo)
    ws = torch.empty(nbytes + 64, dtype=torch.uint8, device="cuda")
    _lib.check(lib.fmb_attn_bwd(*p(do), *p(q), *p(k), *p(v), *p(out), lse.data_ptr(), *p(dq), *p(dk), *p(dv), sd.data_ptr(), co, cn,
                                ind, n_indices, cu.data_ptr(), cu.data_ptr(), ws.data_ptr() + shift, nbytes, *tail, T, mx, mx, chunk,
                                d ** -0.5, 1, 0, stream))
    for a, b in zip((dq, dk, dv), want_grads):
        assert torch.equal(a, b)
