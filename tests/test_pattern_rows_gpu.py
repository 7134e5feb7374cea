"""The pattern builder's row-major view (fmb_build_csc_rows) and its two ways to the tiles' cursors (few tiles:
summed by every scatter CTA; more than 16 tiles of 512 rows: a launch of their own), at the edges of its
512-row tiles, its 1024-column ranges and its list lengths (8, 16, longer).  Everything is exact."""
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


@pytest.mark.parametrize("lens,H,topk,ncol", [
    ([512, 1, 513], 2, 8, 40), ([8192], 1, 8, 64), ([8193, 700, 0, 9000], 2, 3, 1024), ([8200], 1, 16, 1025),
    ([1500], 2, 12, 2100), ([600, 40], 2, 20, 1030), ([9000], 1, 17, 70), ([100], 3, 1, 1),
    ([513, 700], 2, 8, 32), ([513, 700], 2, 8, 33), ([1100], 2, 16, 32), ([1100], 2, 13, 33), ([900], 2, 4, 1030),   # stored by the row, in order
])
def test_row_slots_and_columns(lens, H, topk, ncol):
    from flash_moba_b200 import _lib
    T, mx = sum(lens), max(lens)
    g = torch.Generator().manual_seed(T + topk)
    # distinct ids in random order, a random number of them, empty places anywhere
    idx = torch.rand(T, H, ncol, generator=g).argsort(dim=-1)[..., :topk].to(torch.int32)
    if ncol < topk:
        idx = torch.cat([idx, torch.full((T, H, topk - ncol), -1, dtype=torch.int32)], dim=-1)
    idx[torch.rand(T, H, topk, generator=g) < 0.2] = -1
    cu = cu_of(lens)
    lists, cud = idx.permute(1, 0, 2).contiguous().to(DEV), cu.to(DEV)
    B = len(lens)
    co = torch.empty(B, H, ncol, dtype=torch.int64, device=DEV)
    cn = torch.empty(B, H, ncol, dtype=torch.int32, device=DEV)
    ind = torch.empty(T * H * topk, dtype=torch.int32, device=DEV)
    rows = torch.full((H, T, topk), -7, dtype=torch.int32, device=DEV)
    nbytes = _lib.lib.fmb_build_csc_workspace_bytes(B, H, mx, ncol)
    ws = torch.empty(nbytes, dtype=torch.uint8, device=DEV)
    _lib.check(_lib.lib.fmb_build_csc_rows(lists.data_ptr(), topk, T * topk, cud.data_ptr(), co.data_ptr(), cn.data_ptr(),
                                           ind.data_ptr(), rows.data_ptr(), ws.data_ptr(), nbytes, B, H, topk, T, mx, ncol,
                                           torch.cuda.current_stream().cuda_stream))
    rco, rcn, rind = O.build_csc(idx, cu, topk, ncol)
    assert torch.equal(co.cpu(), rco) and torch.equal(cn.cpu(), rcn) and torch.equal(ind.cpu(), rind)
    slots = rows.cpu().long() & 0xffffffff
    used = slots != 0xffffffff
    count = (idx >= 0).sum(-1).t()                                  # (H, T)
    assert torch.equal(used.sum(-1), count)
    assert (used == (torch.arange(topk).view(1, 1, -1) < count.unsqueeze(-1))).all()      # empty places last
    assert (slots[..., 1:] >= slots[..., :-1]).all() and len(slots[used].unique()) == int(used.sum())
    local = torch.cat([torch.arange(n) for n in lens]).view(1, T, 1).expand(H, T, topk)
    assert torch.equal(rind[slots[used]].long(), local[used])       # every place holds the row it is listed for
    # ... in the column of one of the row's chunks: the columns of a row's places are its list, in order
    seq = torch.cat([torch.full((n,), b) for b, n in enumerate(lens)])
    for h in range(H):
        for t in range(0, T, max(1, T // 50)):
            n = int(count[h, t])
            col = torch.searchsorted(rco[seq[t], h], slots[h, t, :n], right=True) - 1
            while n and (rcn[seq[t], h][col] == 0).any():           # empty columns share the next one's offset
                col = torch.where(rcn[seq[t], h][col] == 0, col - 1, col)
            assert torch.equal(col.int(), idx[t, h][idx[t, h] >= 0].sort().values)


def test_duplicate_ids_count_once():
    from flash_moba_b200 import ops
    idx = torch.tensor([[[3, 3, 1]], [[1, 1, 1]], [[-1, 0, 3]]], dtype=torch.int32)
    once = torch.tensor([[[3, -1, 1]], [[1, -1, -1]], [[-1, 0, 3]]], dtype=torch.int32)
    cu = cu_of([3])
    got = ops.build_csc(idx.permute(1, 0, 2).contiguous().to(DEV).permute(1, 0, 2), cu.to(DEV), 3, 4)
    for a, b in zip(got, O.build_csc(once, cu, 3, 4)):
        assert torch.equal(a.cpu(), b)


@pytest.mark.parametrize("topk", [8, 16])
def test_row_slots_of_any_alignment(topk):
    """row_slots is an array of 32-bit numbers that may start anywhere."""
    from flash_moba_b200 import _lib
    T, H, ncol = 700, 2, 40
    g = torch.Generator().manual_seed(topk)
    lists = torch.rand(H, T, ncol, generator=g).argsort(dim=-1)[..., :topk].to(torch.int32).to(DEV)
    cu = cu_of([T]).to(DEV)
    nbytes = _lib.lib.fmb_build_csc_workspace_bytes(1, H, T, ncol)
    got = []
    for shift in (0, 1, 2, 3):
        co, cn = torch.empty(1, H, ncol, dtype=torch.int64, device=DEV), torch.empty(1, H, ncol, dtype=torch.int32, device=DEV)
        ind, ws = torch.empty(T * H * topk, dtype=torch.int32, device=DEV), torch.empty(nbytes, dtype=torch.uint8, device=DEV)
        rows = torch.full((H * T * topk + 4,), -7, dtype=torch.int32, device=DEV)
        _lib.check(_lib.lib.fmb_build_csc_rows(lists.data_ptr(), topk, T * topk, cu.data_ptr(), co.data_ptr(), cn.data_ptr(),
                                               ind.data_ptr(), rows.data_ptr() + 4 * shift, ws.data_ptr(), nbytes, 1, H, topk, T, T,
                                               ncol, torch.cuda.current_stream().cuda_stream))
        n = H * T * topk
        assert (rows[:shift] == -7).all() and (rows[shift + n:] == -7).all()
        got.append(rows[shift:shift + n].clone())
    assert all(torch.equal(x, got[0]) for x in got)
