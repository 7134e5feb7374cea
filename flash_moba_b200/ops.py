"""Thin PyTorch wrappers over the library, one function per stage; `flash_moba_b200.interface`
composes them into the reference's public API.

The stages' host side (checks, output and workspace allocation from the torch caching allocator, raw
pointers + the current CUDA stream into the C ABI) is native code (csrc/fmb_torch.cpp); the
arithmetic lives entirely in libflashmoba_b200.so.  Nothing here computes on tensors.
"""
import threading as _threading
from typing import Optional, Tuple

import torch

from . import _lib
from ._lib import check, lib, native


def _dtype_code(t: torch.Tensor) -> int:
    if t.dtype == torch.bfloat16:
        return _lib.FMB_BF16
    if t.dtype == torch.float16:
        return _lib.FMB_FP16
    raise RuntimeError("FlashMoBA only supports fp16 and bf16 data type")


def _stream() -> int:
    return torch.cuda.current_stream().cuda_stream


def _require_cuda(*ts):
    for t in ts:
        if t is not None and not t.is_cuda:
            raise RuntimeError("flash_moba_b200: all tensors must be on a CUDA device (there is no CPU path)")


def _i32c(t: torch.Tensor, name: str) -> torch.Tensor:
    if t.dtype != torch.int32:
        raise RuntimeError(f"{name} must have dtype int32")
    if not t.is_contiguous():
        raise RuntimeError(f"{name} must be contiguous")
    return t


def ptr(t: Optional[torch.Tensor]) -> int:
    return 0 if t is None else t.data_ptr()


# ---- the pattern's slot / row lists, handed from a forward call to its backward call
# Both attention calls need the CSR transpose of the pattern in their workspace.  For a pattern the
# library did not build itself attn_fwd keeps a copy of it (a few bytes per pattern entry) that the
# autograd Function collects with take_lists() right after its forward op and offers to the backward
# op with offer_lists(); the custom ops' signatures stay the reference's.  For the library's own
# patterns the builder's row-major view is recognised natively and there is nothing to hand over.
# FMB_SHARE_LISTS=0 turns both off.
_tls = _threading.local()


def _lists_key(col_offsets, col_nnz, indices, cu_seqlens_q, total_q, h, hk, d, batch, max_seqlen_k, chunk):
    """What the lists depend on: the pattern tensors and the sequence bounds (storage and version), the geometry."""
    ident = tuple((t.data_ptr(), 0 if t.is_inference() else t._version, t.numel())
                  for t in (col_offsets, col_nnz, indices, cu_seqlens_q))
    return ident + (int(total_q), h, hk, d, batch, int(max_seqlen_k), int(chunk), str(indices.device))


def take_lists():
    """The lists kept by the last attn_fwd of this thread (None if it kept none); clears the slot."""
    got = getattr(_tls, "kept", None)
    _tls.kept = None
    return got


def offer_lists(lists) -> None:
    """Lists for the next attn_bwd of this thread (used only if they belong to its pattern)."""
    _tls.offered = lists


def check_pending_status() -> None:
    """Waits for the status words of all attention calls issued so far by this process and raises
    for the first one that reports a failure.

    Every attention call leaves a device-side status word: 0, or which bounded wait gave up / 7 = the
    pattern did not fit the slots.  By default the library stores the word into pinned host memory at
    the end of the call, without synchronising, and the attention calls that follow (or this
    function) look at it: a failure raises one call late, never silently.  With FMB_CHECK_STATUS=1
    every call synchronises and raises at once (the tests)."""
    native.check_pending_status()


def selftest_umma(a: torch.Tensor, b: torch.Tensor, b_mn_major: bool) -> torch.Tensor:
    """128x128x128 product on the tcgen05 path (see fmb_selftest_umma)."""
    _require_cuda(a, b)
    a, b = a.contiguous(), b.contiguous()
    with torch.cuda.device(a.device):
        d = torch.empty((128, 128), dtype=torch.float32, device=a.device)
        status = torch.zeros((1,), dtype=torch.int32, device=a.device)
        check(lib.fmb_selftest_umma(ptr(a), ptr(b), ptr(d), int(b_mn_major), _dtype_code(a), ptr(status), _stream()))
        if int(status.item()) != 0:
            raise RuntimeError(f"selftest_umma: bounded wait expired (code {int(status.item())})")
    return d


def selftest_wait_expiry(device=None) -> Tuple[int, float]:
    """Runs the library's bounded wait on an mbarrier nobody arrives at (see fmb_selftest_wait_expiry).
    Returns (status code written by the kernel, seconds the wait lasted before it gave up)."""
    return _expire(lib.fmb_selftest_wait_expiry, device)


def selftest_spin_expiry(device=None) -> Tuple[int, float]:
    """The same of the wait of the threads that issue the backward's MMAs (see fmb_selftest_spin_expiry)."""
    return _expire(lib.fmb_selftest_spin_expiry, device)


def _expire(call, device) -> Tuple[int, float]:
    dev = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    with torch.cuda.device(dev):
        status = torch.full((1,), -1, dtype=torch.int32, device=dev)
        ns = torch.zeros((1,), dtype=torch.int64, device=dev)
        check(call(ptr(status), ptr(ns), _stream()))
        torch.cuda.synchronize(dev)
    return int(status.item()), int(ns.item()) * 1e-9


def set_engine(engine: int) -> int:
    """0 = CUDA-core validation kernels, 1 = tcgen05 kernels.  Returns the engine in use."""
    return lib.fmb_set_engine(int(engine))


# ------------------------------------------------------------------------------- stage P
def mean_pool(k: torch.Tensor, cu_seqlens_k: torch.Tensor, max_seqlen_k: int, chunk: int
              ) -> Tuple[torch.Tensor, torch.Tensor]:
    """Centroids of every chunk.  No host sync: km is allocated with an upper bound of
    ceil(total_k/chunk) + batch rows; rows [0, cu_seqlens_km[-1]) are valid."""
    return native.mean_pool(k, cu_seqlens_k, int(max_seqlen_k), int(chunk))


# ------------------------------------------------------------------------------- stage G
def gate_topk(q, km, cu_seqlens_q, cu_seqlens_k, cu_seqlens_km, max_seqlen_q: int, max_seqlen_k: int,
              topk: int, chunk: int, causal: bool, return_values: bool = False):
    """Per-row top-k chunk lists.  Returns idx as a (total_q, heads, topk) VIEW of a
    head-major (heads, total_q, topk) buffer (the layout the pattern builder streams), and
    the scores in the same layout (or None)."""
    idx, val = native.gate_topk(q, km, cu_seqlens_q, cu_seqlens_k, cu_seqlens_km, int(max_seqlen_q), int(max_seqlen_k),
                                int(topk), int(chunk), bool(causal), return_values)
    return idx.permute(1, 0, 2), (val.permute(1, 0, 2) if val is not None else None)


# --------------------------------------------------------------------------- stages O/E/S
def build_csc(topk_idx: torch.Tensor, cu_seqlens_q: torch.Tensor, max_seqlen_q: int, ncol: int,
              keep_rows: bool = False):
    """(col_offsets i64 (B,H,ncol), col_nnz i32 (B,H,ncol), indices i32 (T*H*topk)).

    keep_rows: also let the library write the pattern's row-major view and keep it for attention
    calls on the returned tensors (only for lists that name a chunk at most once per row, as the
    lists of gate_topk do)."""
    return native.build_csc(topk_idx, cu_seqlens_q, int(max_seqlen_q), int(ncol), keep_rows)


def varlen_sort(starts: torch.Tensor, ends: torch.Tensor, src: torch.Tensor) -> torch.Tensor:
    _require_cuda(starts, ends, src)
    if starts.dtype != torch.int64 or ends.dtype != torch.int64 or src.dtype != torch.int32:
        raise RuntimeError("varlen_sort: offsets must be int64 and keys int32")
    starts, ends, src = starts.contiguous(), ends.contiguous(), src.contiguous()
    with torch.cuda.device(src.device):
        dst = torch.empty_like(src)
        check(lib.fmb_varlen_sort(ptr(starts), ptr(ends), ptr(src), ptr(dst), starts.numel(), src.numel(), _stream()))
    return dst


# ------------------------------------------------------------------------------- stage F
def _key_spans(cu_seqlens_k, leftpad_k, seqused_k, batch):
    """(first key row, one past the last key row) per sequence for the reference's leftpad_k /
    seqused_k arguments (csrc/flash_moba/src/block_info.h:19-26): keys start leftpad_k[b] rows into
    the sequence's storage and seqused_k[b] rows of the storage are in use."""
    for t, n in ((leftpad_k, "leftpad_k"), (seqused_k, "seqused_k")):
        if t is not None:
            _require_cuda(t)
            if tuple(_i32c(t, n).shape) != (batch,):
                raise RuntimeError(f"{n} must have shape (batch_size,)")
    begin = cu_seqlens_k[:-1] if leftpad_k is None else cu_seqlens_k[:-1] + leftpad_k
    end = cu_seqlens_k[1:] if seqused_k is None else cu_seqlens_k[:-1] + seqused_k
    return begin.contiguous(), end.contiguous()


def attn_fwd(q, k, v, col_offsets, col_nnz, indices, cu_seqlens_q, cu_seqlens_k, max_seqlen_q: int,
             max_seqlen_k: int, chunk: int, softmax_scale: float, causal: bool, out: Optional[torch.Tensor] = None,
             leftpad_k: Optional[torch.Tensor] = None, seqused_k: Optional[torch.Tensor] = None):
    """Block-sparse forward.  Returns (out (T,H,d), lse (H,T) fp32)."""
    k_begin = k_end = None
    if leftpad_k is not None or seqused_k is not None:
        k_begin, k_end = _key_spans(_i32c(cu_seqlens_k, "cu_seqlens_k"), leftpad_k, seqused_k, cu_seqlens_q.numel() - 1)
    out, lse, lists = native.attn_fwd(q, k, v, col_offsets, col_nnz, indices, cu_seqlens_q, cu_seqlens_k, int(max_seqlen_q),
                                      int(max_seqlen_k), int(chunk), float(softmax_scale), bool(causal), out, k_begin, k_end)
    _tls.kept = None
    if lists is not None:
        total_q, h, d = q.shape
        _tls.kept = (_lists_key(col_offsets, col_nnz, indices, cu_seqlens_q, total_q, h, k.shape[1], d,
                                cu_seqlens_q.numel() - 1, max_seqlen_k, chunk), lists)
    return out, lse


# ------------------------------------------------------------------------------- stage B
def attn_bwd(dout, q, k, v, out, lse, dq, dk, dv, col_offsets, col_nnz, indices, cu_seqlens_q, cu_seqlens_k,
             max_seqlen_q: int, max_seqlen_k: int, chunk: int, softmax_scale: float, causal: bool) -> torch.Tensor:
    """Block-sparse backward into caller-allocated dq/dk/dv.  Returns softmax_d (H,T) fp32."""
    offered = getattr(_tls, "offered", None)
    _tls.offered = None
    if offered is not None:
        total_q, h, d = q.shape
        mine = _lists_key(col_offsets, col_nnz, indices, cu_seqlens_q, total_q, h, k.shape[1], d,
                          cu_seqlens_q.numel() - 1, max_seqlen_k, chunk)
        offered = offered[1] if offered[0] == mine else None
    return native.attn_bwd(dout, q, k, v, out, lse, dq, dk, dv, col_offsets, col_nnz, indices, cu_seqlens_q, cu_seqlens_k,
                           int(max_seqlen_q), int(max_seqlen_k), int(chunk), float(softmax_scale), bool(causal), offered)
