"""Who counts the pattern's columns: the scatter kernel itself (sequences of one tile of 512 rows, lists of up to 16,
up to 1,024 columns), a kernel ahead of it (up to 16 tiles), that and a scan (more).  Lists that name a chunk several times, and ids that are no
chunk, at the edges of each.  Everything is exact."""
import pytest
import torch

import test_pattern_rows_gpu as rows
from conftest import cu_of
from oracle import moba_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("topk", [3, 8, 13, 16, 17])
@pytest.mark.parametrize("lens,H,ncol", [
    ([512, 1, 0, 300], 2, 32), ([512, 1, 0, 300], 2, 33), ([200], 3, 1), ([512, 40], 2, 1024), ([512, 40], 2, 1025),   # a tile
    ([513, 20], 2, 32), ([1024], 2, 70), ([2048, 700], 2, 40), ([2049], 2, 33), ([8192], 1, 64),                        # several
    ([8193, 600], 1, 40), ([8193, 600], 1, 1030),                                                                       # a scan
])
def test_chunks_named_several_times(lens, H, ncol, topk):
    from flash_moba_b200 import ops
    T, mx = sum(lens), max(lens)
    g = torch.Generator().manual_seed(T + ncol + topk)
    # a few of the chunks (so that most lists repeat some), places without one, ids beyond the last chunk
    few = torch.randint(0, ncol, (T, H, max(2, topk // 2)), generator=g)
    idx = few.gather(2, torch.randint(0, few.shape[2], (T, H, topk), generator=g)).to(torch.int32)
    u = torch.rand(T, H, topk, generator=g)
    idx[u < 0.1] = -1
    idx[u > 0.95] = ncol
    again = (idx.unsqueeze(-1) == idx.unsqueeze(-2)).tril(-1).any(-1)
    once = idx.masked_fill(again | (idx >= ncol), -1)
    got = ops.build_csc(idx.permute(1, 0, 2).contiguous().to(DEV).permute(1, 0, 2), cu_of(lens).to(DEV), mx, ncol)
    for a, b in zip(got, O.build_csc(once, cu_of(lens), topk, ncol)):
        assert torch.equal(a.cpu(), b)


def test_more_sequences_than_sms():
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows.test_row_slots_and_columns([3] * (2 * sms + 1), 2, 8, 5)


@pytest.mark.parametrize("lens,H,topk,ncol", [([512, 0, 37], 3, 8, 40), ([511], 1, 16, 1024), ([200, 512], 2, 13, 33), ([512], 2, 3, 32), ([0, 9], 2, 16, 70)])
def test_row_slots_of_sequences_of_one_tile(lens, H, topk, ncol):
    rows.test_row_slots_and_columns(lens, H, topk, ncol)
