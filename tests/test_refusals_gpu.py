"""Calls that have no meaning here are refused, whichever way their sizes would take them."""
import pytest
import torch

from conftest import cu_of

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("rows,keys", [(2, 600), (4000, 4000)])
def test_forward_mode_is_refused(rows, keys):
    """No forward-mode derivative exists: a dual tensor must not come back as a plain result (2 rows: the decode kernel's
    sizes, 4000: not)."""
    import torch.autograd.forward_ad as fw

    import flash_moba_b200 as F
    from flash_moba_b200 import _lib
    assert _lib.lib.fmb_decode_preferred(rows, keys, 1, 4, 4, 64, keys, 2, 64) == (rows == 2)
    cq, ck = cu_of([rows]).to(DEV), cu_of([keys]).to(DEV)
    q = torch.randn(rows, 4, 64, device=DEV).bfloat16()
    k = torch.randn(keys, 4, 64, device=DEV).bfloat16()
    cache = F.CentroidCache(1, 4, 64, 64, keys)
    cache.update(k, [0, keys], [keys])
    with fw.dual_level():
        for args in ((fw.make_dual(q, torch.ones_like(q)), k, k), (q, fw.make_dual(k, torch.ones_like(k)), k),
                     (q, k, fw.make_dual(k, torch.ones_like(k)))):
            for grad in (True, False):
                with torch.set_grad_enabled(grad):
                    with pytest.raises((RuntimeError, NotImplementedError)):
                        F.flash_moba_varlen_func(*args, cq, ck, rows, keys, 64, 2)
                    with pytest.raises((RuntimeError, NotImplementedError)):
                        cache.attend(*args, cq, ck, rows, keys, 2)
    F.flash_moba_varlen_func(q, k, k, cq, ck, rows, keys, 64, 2)     # without tangents: taken


@pytest.mark.parametrize("H,Hk,d,chunk,heads_first", [(4, 2, 128, 128, False), (4, 2, 64, 64, False), (16, 2, 64, 64, False), (16, 2, 64, 64, True)])
def test_rows_that_span_more_than_64_gib(H, Hk, d, chunk, heads_first):
    """A view of rows that lie far apart: offsets of more than 2^32 units of 16 bytes (16 / 2 heads: items of several heads)."""
    import flash_moba_b200 as F
    if torch.cuda.mem_get_info()[0] < 100 << 30:
        pytest.skip("needs 100 GiB of free device memory")
    lens, topk = ([1500], 3) if H == 4 else ([63] * 160 + [200] * 5, 2)
    T = sum(lens)
    torch.manual_seed(d)
    base = torch.randn(T, H, d, device=DEV).bfloat16()
    k, v = (torch.randn(T, Hk, d, device=DEV).bfloat16() for _ in range(2))
    elements = 36 << 30                                         # 72 GiB
    buf = torch.empty(elements, dtype=torch.bfloat16, device=DEV)
    try:
        rs = (elements - H * d) // T // d * d
        q = buf.as_strided((T, H, d), (d, elements // H // d * d, 1) if heads_first else (rs, d, 1))
        assert heads_first or (T - 1) * rs * 2 > 64 << 30
        q.copy_(base)
        cu = cu_of(lens).to(DEV)
        with torch.no_grad():
            pattern = F.flash_topk_varlen_func(base, k, cu, cu, max(lens), max(lens), topk, chunk, causal=True)
            args = (k, v, cu, cu, max(lens), max(lens), *pattern, 128, chunk)
            want = F.flash_moba_attn_varlen_func(base, *args, causal=True, return_attn_probs=True)
            got = F.flash_moba_attn_varlen_func(q, *args, causal=True, return_attn_probs=True)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
        got = None
        from flash_moba_b200 import ops
        do = torch.randn(T, H, d, device=DEV).bfloat16()
        grads = []
        for x in (base, q):
            g = [torch.empty_like(t) for t in (base, k, v)]
            ops.attn_bwd(do, x, k, v, want[0], want[1], *g, *pattern, cu, cu, max(lens), max(lens), chunk, d ** -0.5, True)
            grads.append(g)
        assert all(torch.equal(a, b) for a, b in zip(*grads))
    finally:
        x = q = buf = args = None
        torch.cuda.empty_cache()


def test_rows_whose_distance_fits_no_unit():
    """More than 64 GiB apart and no multiple of a head's row: the CUDA-core kernels take the call.  Both engines round
    probabilities and partial results to 8 bits, at most 2^-8 each of sums of topk parts: 1e-2 in the 2-norm."""
    import flash_moba_b200 as F
    if torch.cuda.mem_get_info()[0] < 100 << 30:
        pytest.skip("needs 100 GiB of free device memory")
    T, H, d, chunk = 1500, 4, 64, 64
    torch.manual_seed(5)
    base = torch.randn(T, H, d, device=DEV).bfloat16()
    k, v = (torch.randn(T, 2, d, device=DEV).bfloat16() for _ in range(2))
    buf = torch.empty(36 << 30, dtype=torch.bfloat16, device=DEV)
    try:
        q = buf.as_strided((T, H, d), (((36 << 30) - H * d) // T // 8 * 8 // 64 * 64 + 8 - 64, d, 1))
        q.copy_(base)
        cu = cu_of([T]).to(DEV)
        with torch.no_grad():
            pattern = F.flash_topk_varlen_func(base, k, cu, cu, T, T, 3, chunk, causal=True)
            want, got = (F.flash_moba_attn_varlen_func(x, k, v, cu, cu, T, T, *pattern, 128, chunk, causal=True).float() for x in (base, q))
        assert (got - want).norm() <= 1e-2 * want.norm()
    finally:
        q = buf = None
        torch.cuda.empty_cache()


def test_a_launch_that_fails_leaves_no_error_behind():
    """The runtime keeps a thread's last error until it is asked for: a refused call must not make the next one, of this library or
    of torch, report it.  (More column groups than a grid may have: the runtime refuses the launch, nothing runs.)"""
    import ctypes

    from flash_moba_b200 import _lib, ops
    cudart = ctypes.CDLL("libcudart.so.12")
    some = torch.zeros(4096, dtype=torch.int64, device=DEV)
    ncol = 8192 * 65536                                  # 65536 groups of the histogram's 8192 columns
    rc = _lib.lib.fmb_build_csc(*[some.data_ptr(), 1, 1] + [some.data_ptr()] * 5, 4 * ncol + 256, 1, 1, 1, 16, ncol,
                                torch.cuda.current_stream().cuda_stream)
    assert rc != 0
    assert cudart.cudaPeekAtLastError() == 0
    assert b"csc_tile_hist_kernel" in _lib.lib.fmb_last_error()
    k = torch.ones(100, 2, 64, device=DEV, dtype=torch.bfloat16)
    km, _ = ops.mean_pool(k, torch.tensor([0, 100], dtype=torch.int32, device=DEV), 100, 64)
    assert (km[:2] == 1).all()
