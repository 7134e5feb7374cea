"""Calls in the middle of other work: inputs that the kernel just before writes, inputs and results that the kernel just behind
overwrites, one call on the tail of another, and all of it as a CUDA graph.  Kernels of a call are brought up while the one
before still runs, so a wait too few would show here.  Same bits as the same call with the device idle around it."""
import pytest
import torch

from conftest import cu_of

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _inputs(lens_q, lens_k, H, Hk, d, seed):
    g = torch.Generator().manual_seed(seed)
    return [torch.randn(n, h, d, generator=g).bfloat16().to(DEV)
            for n, h in ((sum(lens_q), H), (sum(lens_k), Hk), (sum(lens_k), Hk), (sum(lens_q), H))]


def _between_writers(sets, call, monkeypatch):
    """`call(buffers, source)` alone on each of the sets, then on one set of buffers that is filled just before and overwritten just
    behind, then as a graph."""
    monkeypatch.setenv("FMB_CHECK_STATUS", "0")          # (no synchronisation inside a call)
    want = []
    for s in sets:
        bufs = [t.clone() for t in s]
        torch.cuda.synchronize()
        want.append([t.clone() for t in call(bufs, s)])
        torch.cuda.synchronize()
    bufs = [torch.full_like(t, float("nan")) for t in sets[0]]
    got = []

    def turn(s):
        for b, t in zip(bufs, s):
            b.copy_(t)
        out = call(bufs, s)
        for b in bufs:
            b.fill_(float("nan"))
        kept = [t.clone() for t in out]
        for t in out:
            t.fill_(float("nan"))
        return kept

    for i in range(6):
        got.append(turn(sets[i % 2]))
    torch.cuda.synchronize()
    for i, outs in enumerate(got):
        for a, b in zip(outs, want[i % 2]):
            assert torch.equal(a, b), i
    source = [t.clone() for t in sets[0]]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        turn(source)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outs = turn(source)
        again = turn(source)                             # one call on the tail of the other inside the graph
    for i in range(4):
        for t, s in zip(source, sets[i % 2]):
            t.copy_(s)
        graph.replay()
        for a, b, w in zip(outs, again, want[i % 2]):
            assert torch.equal(a, w) and torch.equal(b, w), i


@pytest.mark.parametrize("lens,H,Hk,d,chunk,topk", [
    ([900, 515], 8, 2, 128, 128, 4),
    ([700, 260, 33], 12, 12, 64, 64, 8),
    ([700, 260], 6, 6, 64, 128, 3),
    ([9000], 4, 2, 128, 64, 16),                         # counts of the pattern scanned by a kernel of their own
    ([600, 200], 4, 4, 256, 64, 3),
])
def test_training_step(lens, H, Hk, d, chunk, topk, monkeypatch):
    import flash_moba_b200 as F
    cu = cu_of(lens).to(DEV)

    def call(bufs, source):
        q, k, v, do = bufs
        leaves = [t.detach().requires_grad_(True) for t in (q, k, v)]
        out = F.flash_moba_varlen_func(*leaves, cu, cu, max(lens), max(lens), chunk, topk, causal=True)
        do.fill_(float("nan"))
        do.copy_(source[3])                              # the gradient is written just before the backward pass reads it
        return [out.detach()] + list(torch.autograd.grad(out, leaves, do))

    _between_writers([_inputs(lens, lens, H, Hk, d, s) for s in (1, 2)], call, monkeypatch)


@pytest.mark.parametrize("cached", [False, True])
@pytest.mark.parametrize("lens_k,H,Hk,d", [
    ([6001], 32, 8, 128),                                # clusters of eight CTAs
    ([3000, 2500, 2001, 777], 32, 8, 128),               # of four
    ([2000 + 37 * i for i in range(16)], 32, 8, 128),    # of two
    ([900 + 37 * i for i in range(40)], 16, 16, 64),
])
def test_decoding_step(lens_k, H, Hk, d, cached, monkeypatch):
    """Without a cache of centroids the pool kernel runs just before the decode kernel; with one, the keys' last writer does."""
    import flash_moba_b200 as F
    from flash_moba_b200 import _lib
    chunk, topk, n = 128, 8, len(lens_k)
    lens_q = [1] * n
    cq, ck, mk = cu_of(lens_q).to(DEV), cu_of(lens_k).to(DEV), max(lens_k)
    assert _lib.lib.fmb_decode_preferred(n, sum(lens_k), n, H, Hk, d, mk, topk, chunk)
    offsets = [0] + torch.tensor(lens_k).cumsum(0).tolist()
    sets = [_inputs(lens_q, lens_k, H, Hk, d, s) for s in (1, 2)]
    if cached:                                           # centroids are of the first set in every turn
        cache = F.CentroidCache(n, Hk, d, chunk, mk, dtype=torch.bfloat16)
        cache.update(sets[0][1], offsets, lens_k)

    def call(bufs, source):
        q, k, v, _ = bufs
        with torch.no_grad():
            if cached:
                return [cache.attend(q, k, v, cq, ck, 1, mk, topk)]
            return [F.flash_moba_varlen_func(q, k, v, cq, ck, 1, mk, chunk, topk, causal=True)]

    _between_writers(sets, call, monkeypatch)
