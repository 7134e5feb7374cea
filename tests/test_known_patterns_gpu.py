"""Patterns of the library's own builder that come back through flash_moba_attn_varlen_func: the row-major view kept beside them
is used only where it describes the call, lives as long as a kernel may read it, and is not part of what autograd
saves.  The checker is the same call on copies of the pattern tensors, for which the library builds its own lists."""
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
