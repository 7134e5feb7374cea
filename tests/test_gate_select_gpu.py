"""The two-sweep gating kernel at the sizes where it can go wrong: candidate counts around its 64-column
score tiles and the four tiles that stay in TMEM, many tiles, lists shorter than the kernel's 8 or 16
places, masses of equal scores (its queues run full), rows without candidates, ragged row tiles.

Integer-valued queries and centroids make every fp32 score exact, so the lists must equal the oracle's
entry by entry, ties (the higher chunk id first) included."""
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


@pytest.mark.parametrize("spread", [0, 1, 6])       # 0: every score is the same
@pytest.mark.parametrize("lens_q,lens_k,H,Hk,d,topk,causal", [
    ([130], [130], 2, 2, 64, 8, True),              # candidates 0 ... 129: one to three tiles, two row tiles
    ([1, 63, 64], [65, 128, 256], 4, 2, 128, 5, True),
    ([128], [257], 2, 1, 128, 8, False),            # five tiles: the products are computed twice
    ([20, 7], [256, 255], 2, 2, 128, 16, False),    # four tiles, lists of 16
    ([40], [1500], 2, 1, 64, 11, True),             # 24 tiles, lists of 11
    ([3, 0, 30], [640, 10, 2111], 2, 2, 128, 1, True),
    ([9], [700], 2, 2, 256, 13, False),
    ([50], [20], 2, 2, 64, 4, True),                # more rows than keys
    ([2] * 70, [90 + i for i in range(70)], 6, 2, 96, 7, True),   # more sequences than are kept in shared memory
])
def test_gate_select_exact(lens_q, lens_k, H, Hk, d, topk, causal, spread):
    from flash_moba_b200 import ops
    g = torch.Generator().manual_seed(d + topk)
    q = torch.randint(-2, 3, (sum(lens_q), H, d), generator=g).to(torch.bfloat16) if spread else torch.ones(sum(lens_q), H, d).bfloat16()
    km = torch.randint(-spread, spread + 1, (sum(lens_k), Hk, d), generator=g).to(torch.bfloat16)
    cq, ck = cu_of(lens_q), cu_of(lens_k)            # chunks of one key: the centroids are the keys
    for values in (True, False):
        idx, val = ops.gate_topk(q.to(DEV), km.to(DEV), cq.to(DEV), ck.to(DEV), ck.to(DEV), max(lens_q), max(lens_k), topk, 1,
                                 causal, return_values=values)
        ref_idx, ref_val = O.gate_topk(q, km, cq, ck, ck, topk, 1, causal)
        assert torch.equal(idx.cpu(), ref_idx)
        assert val is None or torch.equal(val.cpu(), ref_val)


@pytest.mark.parametrize("topk,causal,n_values", [(8, True, 400), (8, False, 400), (16, True, 300), (16, False, 60), (5, True, 40), (12, False, 500), (8, True, 12), (16, True, 20)])
def test_scores_that_differ_in_their_last_bits(topk, causal, n_values):
    """Lists are put in order by the upper 26 bits of the scores first.  Here a score is an integer of six or seven bits plus 0 to 3 times
    2**-15, exact in fp32: among the integers' repetitions are equal scores, pairs that differ below those bits, and more than two of a kind."""
    from flash_moba_b200 import ops
    g = torch.Generator().manual_seed(topk + n_values)
    lens_q, lens_k, H, Hk, d = [200, 77], [260, 333], 2, 1, 128
    q = torch.zeros(sum(lens_q), H, d)
    q[..., 0], q[..., 5] = 1.0, 2.0 ** -15
    sign = torch.randint(0, 2, (sum(lens_q), H), generator=g) * 2 - 1
    q[..., 0] *= sign
    km = torch.zeros(sum(lens_k), Hk, d)
    # (an integer of up to eight bits is exact in bf16)
    km[..., 0] = torch.randint(0, n_values, (sum(lens_k), Hk), generator=g).remainder(127).float() + 1
    km[..., 5] = torch.randint(0, 4, (sum(lens_k), Hk), generator=g).float()
    q, km = q.bfloat16(), km.bfloat16()
    cq, ck = cu_of(lens_q), cu_of(lens_k)
    idx, val = ops.gate_topk(q.to(DEV), km.to(DEV), cq.to(DEV), ck.to(DEV), ck.to(DEV), max(lens_q), max(lens_k), topk, 1, causal,
                             return_values=True)
    ref_idx, ref_val = O.gate_topk(q, km, cq, ck, ck, topk, 1, causal)
    assert torch.equal(idx.cpu(), ref_idx) and torch.equal(val.cpu(), ref_val)


def _scores(kind, n, rng):
    """Integer scores of n candidates, exact in bf16."""
    if kind == "equal":
        return torch.full((n,), 3.0)
    if kind == "ascending":                          # block by block of 16
        return (torch.arange(n) // 16).float()
    if kind == "smooth":                             # neighbouring chunks score alike, few values
        return torch.randint(-1, 2, (n,), generator=rng).cumsum(0).clamp(-200, 200).float()
    assert kind == "one share"                       # the best are all in the columns of one of a row's two threads
    best = torch.arange(n) % 32 < 16
    return torch.where(best, torch.randint(60, 64, (n,), generator=rng), torch.randint(0, 50, (n,), generator=rng)).float()


@pytest.mark.parametrize("kind", ["equal", "ascending", "smooth", "one share"])
@pytest.mark.parametrize("d,topk,causal,lens_k", [
    (128, 16, False, [36, 700]), (64, 16, False, [65, 256]), (256, 16, False, [257, 300]),
    (128, 16, False, [600, 320]), (128, 15, False, [129, 420]), (128, 16, True, [700, 300]),
    (128, 8, False, [40, 610]), (64, 8, True, [300, 200]), (128, 9, False, [500, 64]),
])
def test_queues_that_run_full(kind, d, topk, causal, lens_k):
    """More candidates than a queue has room for, in row tiles whose 128 rows all have some, so that every warp pair's queues are in use:
    zero and repeated keys, padding rows, scores that are smooth from chunk to chunk.  The lists are the oracle's, each time."""
    from flash_moba_b200 import ops
    g = torch.Generator().manual_seed(d + topk + lens_k[0])
    lens_q, H, Hk = [200, 130], 4, 2
    q = torch.zeros(sum(lens_q), H, d)
    q[..., 3] = torch.randint(0, 2, (sum(lens_q), H), generator=g).float() * 2 - 1      # the scores, or their negatives
    q[torch.rand(sum(lens_q), generator=g) < 0.2] = 0.0                                 # rows without any preference
    km = torch.zeros(sum(lens_k), Hk, d)
    at = 0
    for n in lens_k:
        for h in range(Hk):
            km[at:at + n, h, 3] = _scores(kind, n, g)
        at += n
    q, km = q.bfloat16(), km.bfloat16()
    cq, ck = cu_of(lens_q), cu_of(lens_k)
    ref_idx, ref_val = O.gate_topk(q, km, cq, ck, ck, topk, 1, causal)
    for _ in range(3):
        idx, val = ops.gate_topk(q.to(DEV), km.to(DEV), cq.to(DEV), ck.to(DEV), ck.to(DEV), max(lens_q), max(lens_k), topk, 1, causal,
                                 return_values=True)
        assert torch.equal(idx.cpu(), ref_idx) and torch.equal(val.cpu(), ref_val)
