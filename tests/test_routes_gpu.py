"""Which way a call takes, and that every way gives the oracle's result: CentroidCache.attend below the size rule of the decode
kernel (fmb_decode_preferred) and above it, the public function likewise, and the gating entry point without sizes,
which runs another kernel than the one with sizes."""
import pytest
import torch

from conftest import cu_of
from test_gate_select_gpu import O, test_gate_select_exact as sized

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _oracle(q, k, v, km, cu_km, cq, ck, topk, chunk):
    idx, _ = O.gate_topk(q, km, cq, ck, cu_km, topk, chunk, True)
    return O.attention_blocked(q.float(), k.float(), v.float(), cq, ck, idx, chunk, True)[0], idx


@pytest.mark.parametrize("cached", [True, False])
@pytest.mark.parametrize("lens_q,lens_k,H,Hk,d,chunk,topk,decode", [
    ([1, 1], [700, 333], 8, 2, 128, 128, 3, True),
    ([4, 1, 9], [2000, 65, 300], 4, 4, 64, 64, 4, True),
    ([1], [900], 4, 1, 256, 128, 3, True),
    ([700, 1, 1000], [900, 2000, 1000], 8, 2, 128, 128, 3, False),       # blocks of new rows behind their caches
    ([600, 900], [700, 900], 16, 4, 64, 64, 5, False),
    ([900], [1500], 8, 2, 256, 128, 2, False),
    ([700], [1100], 12, 4, 96, 64, 3, False),                            # between the built head dims: padded
])
def test_attend_against_the_oracle(lens_q, lens_k, H, Hk, d, chunk, topk, decode, cached):
    """Tolerance: the fp32 result on the same lists, inputs of 8 significant bits.  The decode kernel rounds only its result
    (2^-8 of the value).  The general path also rounds the probabilities and every chunk's part of a row, at most 2^-8
    each, of sums of up to topk such parts; values are below 6, so that 3 x 2^-8 x 6 = 0.07 bounds each element, and the
    2-norm error of independent roundings (three of 2^-9 on average) is below 4 x 2^-9.  A row whose k-th and (k+1)-th scores
    agree to the last bits of the fp32 sums may select the other chunk: at most one row-head in 200."""
    import flash_moba_b200 as F
    from flash_moba_b200 import _lib
    g = torch.Generator().manual_seed(d + chunk)
    q, k, v = (torch.randn(n, h, d, generator=g).bfloat16() for n, h in ((sum(lens_q), H), (sum(lens_k), Hk), (sum(lens_k), Hk)))
    cq, ck, mq, mk = cu_of(lens_q), cu_of(lens_k), max(lens_q), max(lens_k)
    assert _lib.lib.fmb_decode_preferred(sum(lens_q), sum(lens_k), len(lens_k), H, Hk, d, mk, topk, chunk) == int(decode)
    km, cu_km = O.mean_pool(k, ck, chunk)
    want, _ = _oracle(q, k, v, km, cu_km, cq, ck, topk, chunk)
    dev = [t.to(DEV) for t in (q, k, v)]
    with torch.no_grad():
        if cached:
            cache = F.CentroidCache(len(lens_k), Hk, d, chunk, mk)
            cache.update(dev[1], ck, lens_k)
            got = cache.attend(*dev, cq.to(DEV), ck.to(DEV), mq, mk, topk)
        else:
            got = F.flash_moba_varlen_func(*dev, cq.to(DEV), ck.to(DEV), mq, mk, chunk, topk)
    err = (got.cpu().float() - want).abs()
    bound = 2.0 ** -8 * want.abs() + 1e-3 if decode else torch.full_like(want, 0.07)
    off = (err > bound).any(-1)
    assert off.float().mean() <= 0.005, off.float().mean()
    same = ~off
    assert err[same].norm() <= 4 * 2.0 ** -9 * want[same].norm()


@pytest.mark.parametrize("case", range(9))
@pytest.mark.parametrize("spread", [0, 1, 6])
def test_gating_entry_without_sizes(case, spread):
    """fmb_gate_topk on the cases of the entry with sizes: the lists are the oracle's, entry by entry."""
    from flash_moba_b200 import _lib
    cases = next(m for m in sized.pytestmark if m.name == "parametrize" and "lens_q" in m.args[0]).args[1]
    assert len(cases) == 9
    lens_q, lens_k, H, Hk, d, topk, causal = cases[case]
    g = torch.Generator().manual_seed(d + topk)
    q = torch.randint(-2, 3, (sum(lens_q), H, d), generator=g).bfloat16() if spread else torch.ones(sum(lens_q), H, d).bfloat16()
    km = torch.randint(-spread, spread + 1, (sum(lens_k), Hk, d), generator=g).bfloat16()
    cq, ck = cu_of(lens_q), cu_of(lens_k)
    T = sum(lens_q)
    qd, kd, cqd, ckd = (t.to(DEV) for t in (q, km, cq, ck))
    idx = torch.full((H, T, topk), -5, dtype=torch.int32, device=DEV)
    val = torch.empty((H, T, topk), dtype=torch.float32, device=DEV)
    _lib.check(_lib.lib.fmb_gate_topk(qd.data_ptr(), qd.stride(0), qd.stride(1), kd.data_ptr(), cqd.data_ptr(), ckd.data_ptr(), ckd.data_ptr(),
                                      idx.data_ptr(), val.data_ptr(), topk, T * topk, len(lens_q), H, Hk, d, max(lens_q), max(lens_k),
                                      topk, 1, int(causal), 0, torch.cuda.current_stream().cuda_stream))
    ref_idx, ref_val = O.gate_topk(q, km, cq, ck, ck, topk, 1, causal)
    assert torch.equal(idx.permute(1, 0, 2).cpu(), ref_idx)
    assert torch.equal(val.permute(1, 0, 2).cpu(), ref_val)
