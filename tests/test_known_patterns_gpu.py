"""Patterns of the library's own builder that come back through flash_moba_attn_varlen_func: the row-major view kept beside them
is used only where it describes the call, lives as long as a kernel may read it, and is not part of what autograd
saves.  Compared with the same call on copies of the pattern tensors, for which the library builds its own lists."""
import pytest
import torch

from conftest import cu_of

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _inputs(lens, H=4, Hk=2, d=64, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return [torch.randn(sum(lens), h, d, generator=g, device=DEV).bfloat16() for h in (H, Hk, Hk)]


def _attend(q, k, v, cu, mx, pattern, chunk=64):
    import flash_moba_b200 as F
    return F.flash_moba_attn_varlen_func(q, k, v, cu, cu, mx, mx, *pattern, 128, chunk, causal=True)


def _pattern(q, k, cu, mx, topk=3, chunk=64):
    import flash_moba_b200 as F
    return F.flash_topk_varlen_func(q, k, cu, cu, mx, mx, topk, chunk, causal=True)


def _copies(pattern):
    return tuple(t.clone() for t in pattern)


def test_edit_in_inference_mode():
    lens = [700, 130]
    q, k, v = _inputs(lens)
    cu = cu_of(lens).to(DEV)
    with torch.inference_mode():
        pattern = _pattern(q, k, cu, max(lens))
        pattern[1][:, :, 1] = 0                   # chunk 1 is dropped
        got = _attend(q, k, v, cu, max(lens), pattern)
        want = _attend(q, k, v, cu, max(lens), _copies(pattern))
    assert torch.equal(got, want)


@pytest.mark.parametrize("inference", [False, True])
def test_other_sequence_bounds(inference):
    lens, other = [300, 340], [340, 300]
    q, k, v = _inputs(lens)
    cu, cu2 = cu_of(lens).to(DEV), cu_of(other).to(DEV)
    with torch.inference_mode(inference):
        pattern = _pattern(q, k, cu, 340)
        got = _attend(q, k, v, cu2, 340, pattern)
        want = _attend(q, k, v, cu2, 340, _copies(pattern))
    assert torch.equal(got, want)


def test_bounds_edited_in_place():
    lens = [300, 340]
    q, k, v = _inputs(lens)
    cu = cu_of(lens).to(DEV)
    pattern = _pattern(q, k, cu, 340)
    cu[1] = 340
    assert torch.equal(_attend(q, k, v, cu, 340, pattern), _attend(q, k, v, cu, 340, _copies(pattern)))


def test_rows_used_on_another_stream(monkeypatch):
    """The hidden rows stay what they are until the call that reads them is through, whatever the builder's stream does."""
    monkeypatch.setenv("FMB_CHECK_STATUS", "0")   # (reading the status word back synchronises)
    lens = [3000, 1130]
    q, k, v = _inputs(lens, H=8, Hk=8)
    cu = cu_of(lens).to(DEV)
    want = _attend(q, k, v, cu, max(lens), _copies(_pattern(q, k, cu, max(lens))))
    _pattern(-q, k, cu, max(lens)), torch.full((9,), -1, dtype=torch.int32, device=DEV)   # (loading a kernel waits for the GPU)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    pattern = _pattern(q, k, cu, max(lens))
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        torch.cuda._sleep(2_000_000_000)          # about a second
        got = _attend(q, k, v, cu, max(lens), pattern)
    size = pattern[2].numel()
    for t in pattern:
        t.record_stream(side)                     # as the caller of a second stream does
    del pattern, t
    later = [_pattern(-q, k, cu, max(lens)) for _ in range(5)]
    junk = [torch.full((size,), -1, dtype=torch.int32, device=DEV) for _ in range(16)]
    torch.cuda.synchronize()
    assert torch.equal(got, want) and len(later) + len(junk) == 21


def test_rows_used_under_capture(monkeypatch):
    """A graph that reads the rows of a pattern built before the capture: they live as long as the pattern does."""
    lens = [700, 130]
    q, k, v = _inputs(lens)
    cu = cu_of(lens).to(DEV)
    want = _attend(q, k, v, cu, max(lens), _copies(_pattern(q, k, cu, max(lens))))
    pattern = _pattern(q, k, cu, max(lens))
    _attend(q, k, v, cu, max(lens), pattern)      # warm-up
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    monkeypatch.setenv("FMB_CHECK_STATUS", "0")   # (reading the status word back synchronises)
    with torch.cuda.graph(graph):
        got = _attend(q, k, v, cu, max(lens), pattern)
    later = [_pattern(q, k, cu, max(lens)) for _ in range(6)]
    junk = [torch.full((pattern[2].numel(),), -1, dtype=torch.int32, device=DEV) for _ in range(16)]
    got.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want) and len(later) + len(junk) == 22


def test_a_refused_call_leaves_nothing_behind():
    """Rows handed to a call that fails must not reach the next one."""
    from flash_moba_b200 import _lib
    lens = [700, 130]
    q, k, v = _inputs(lens)
    cu = cu_of(lens).to(DEV)
    pattern = _pattern(q, k, cu, max(lens))
    other = _copies(_pattern(k.repeat(1, 2, 1), k, cu, max(lens)))
    want = _attend(q, k, v, cu, max(lens), other)
    # a batched tensor has no storage: the call fails between the hand-over and the launch
    with pytest.raises(RuntimeError):
        torch.vmap(lambda x: _attend(x, k, v, cu, max(lens), pattern))(q.unsqueeze(0))
    assert torch.equal(_attend(q, k, v, cu, max(lens), other), want)
    # the C entry points: refused for its chunk size
    rows = torch.full((q.shape[1] * q.shape[0] * 3,), -1, dtype=torch.int32, device=DEV)
    for name in ("fmb_attn_fwd", "fmb_attn_bwd"):
        _lib.check(_lib.lib.fmb_attn_rows_offer(rows.data_ptr(), q.shape[0], q.shape[1], 3))
        zeros = [0] * (len(_lib._SIGS[name][1]))
        assert getattr(_lib.lib, name)(*zeros) != 0
        assert torch.equal(_attend(q, k, v, cu, max(lens), other), want), name


def test_checkpointed_layers():
    """Recomputation saves what the first pass saved, however many patterns were built in between."""
    from torch.utils.checkpoint import checkpoint
    lens, layers = [700, 130], 7
    cu = cu_of(lens).to(DEV)
    q, k, v = (t.requires_grad_(True) for t in _inputs(lens))
    patterns = [_pattern(q.detach() * (i + 1), k.detach(), cu, max(lens), topk=2 + i % 3) for i in range(layers)]

    def run(attend):
        out = sum(attend(q, k, v, cu, max(lens), p) for p in patterns)
        return torch.autograd.grad(out, (q, k, v), torch.ones_like(out))

    want = run(_attend)

    def recomputed(q, k, v, cu, mx, p):
        fresh = _pattern(q.detach(), k.detach(), cu, mx)      # a pattern of the layer's own, built again with it
        return checkpoint(lambda q, k, v: _attend(q, k, v, cu, mx, p) + 0 * _attend(q, k, v, cu, mx, fresh), q, k, v, use_reentrant=False)

    for a, b in zip(want, run(recomputed)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("lens,H,Hk,d,chunk,topk", [
    ([1], 3, 1, 128, 128, 1),                     # three rows of one place in all: most warps have none
    ([5, 0, 2], 2400, 2400, 128, 64, 8),          # a warp's next row is hundreds of heads further, three turns of 148 SMs
    ([70, 0, 201], 300, 300, 128, 64, 8),         # eleven turns, rows of one to four places
    ([517], 8, 2, 256, 128, 7),
    ([130, 259], 6, 6, 128, 128, 8),
    ([400], 4, 4, 128, 256, 4),                   # two planes: not staged
    ([300], 4, 4, 128, 64, 9),                    # nine places: not staged
])
def test_rows_merged_from_their_own_lists(lens, H, Hk, d, chunk, topk):
    """The merge of the builder's lists (up to eight places: O staged in shared memory, dQ not for so few partials) against that of
    lists the call builds itself, bit for bit: same partials, same order of the sums.  Rows of no sequence (q is longer than its
    sequences) included."""
    import flash_moba_b200 as F
    q, k, v = _inputs(lens, H, Hk, d, seed=len(lens) + topk)
    pad = torch.randn(3, H, d, device=DEV).bfloat16()
    q = torch.cat([q, pad])
    cu, mx = cu_of(lens).to(DEV), max(lens)
    outs = []
    for copies in (False, True):
        x = [t.detach().clone().requires_grad_(True) for t in (q, k, v)]
        pattern = F.flash_topk_varlen_func(x[0].detach(), x[1].detach(), cu, cu, mx, mx, topk, chunk, causal=True)
        o = F.flash_moba_attn_varlen_func(*x, cu, cu, mx, mx, *(_copies(pattern) if copies else pattern), 128, chunk, causal=True)
        outs.append((o,) + torch.autograd.grad(o, x, torch.ones_like(o)))
    for a, b in zip(*outs):
        assert torch.isfinite(a).all() and torch.equal(a, b)


@pytest.mark.parametrize("lens,H,Hk,d,topk", [
    ([8189], 32, 8, 128, 8),                      # the fewest partials whose dQ is staged: 512 MiB, three rows of no sequence
    ([2500, 1, 4099, 2000], 32, 8, 128, 8),
    ([4701], 32, 4, 256, 7),
])
def test_dq_merged_from_its_own_lists(lens, H, Hk, d, topk):
    """As above where there are enough partials for dQ's merge to be staged too."""
    import flash_moba_b200 as F
    assert (sum(lens) + 3) * H * topk * d * 2 >= 1 << 29
    q, k, v = _inputs(lens, H, Hk, d, seed=d)
    q = torch.cat([q, torch.randn(3, H, d, device=DEV).bfloat16()])
    cu, mx = cu_of(lens).to(DEV), max(lens)
    outs = []
    for copies in (False, True):
        x = [t.detach().clone().requires_grad_(True) for t in (q, k, v)]
        pattern = F.flash_topk_varlen_func(x[0].detach(), x[1].detach(), cu, cu, mx, mx, topk, 128, causal=True)
        o = F.flash_moba_attn_varlen_func(*x, cu, cu, mx, mx, *(_copies(pattern) if copies else pattern), 128, 128, causal=True)
        outs.append((o,) + torch.autograd.grad(o, x, torch.ones_like(o)))
    for a, b in zip(*outs):
        assert torch.isfinite(a).all() and torch.equal(a, b)
