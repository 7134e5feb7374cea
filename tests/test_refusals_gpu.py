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
