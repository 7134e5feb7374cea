"""The forward kernel's ring of item descriptions against the roles that read it: the waits of the kernel as rules over
counts, one reader held up as long as they allow while everyone else goes on, and how far the scout publishes
meanwhile.  (A ring that is too short shows on a GPU only if a warp is late by several GEMMs.)"""
import os
import random
import re

import pytest

from conftest import ROOT

SOURCE = open(os.path.join(ROOT, "flash_moba_b200", "csrc", "fmb_attn_tc.cu")).read()


def _constant(name):
    return int(re.search(r"constexpr int %s = (\d+);" % name, SOURCE).group(1))


def _published_while(role, held, tiles_of, NK, NB, G):
    """Last item published while `role` never gets past tile (V: item) `held`."""
    item = [i for i, n in enumerate(tiles_of) for _ in range(n)]
    last = [i + 1 == len(item) or item[i + 1] != item[i] for i in range(len(item))]
    end = {i: t for t, i in enumerate(item)}              # an item's last tile
    T, N = len(item), len(tiles_of)
    pub, kst, vst = [False] * N, [False] * N, [False] * N
    full, S, ready, PV, tfree, done = ([False] * T for _ in range(6))
    pub[0] = True
    moved = True
    while moved:
        moved = False

        def step(a, i, cond):
            nonlocal moved
            if not a[i] and cond:
                a[i] = moved = True

        for n in range(N):
            step(kst, n, pub[n] and (n < NK or S[end[n - NK]]))
            if n + 1 < N:
                step(pub, n + 1, kst[n])
            step(vst, n, pub[n] and (n == 0 or (vst[n - 1] and PV[end[n - 1]])) and not (role == "v" and n > held))
        for t in range(T):
            prev = t < G
            step(full, t, pub[item[t]] and (prev or full[t - G]) and (t < NB or (full[t - NB] and PV[t - NB]))
                 and not (role == "loader" and t > held and (t - held) % G == 0))
            step(S, t, kst[item[t]] and full[t] and (t == 0 or S[t - 1]) and (prev or tfree[t - G]))
            step(ready, t, S[t] and (prev or done[t - G]))
            step(PV, t, ready[t] and vst[item[t]] and (t == 0 or PV[t - 1]))
            step(tfree, t, PV[t])
            step(done, t, tfree[t] and not (role == "group" and t == held))
    assert last[-1]
    # the held reader has the items behind its own still to look up
    first_needed = (held if role == "v" else item[held]) + 1
    return max(i for i in range(N) if pub[i]) - first_needed + 1


@pytest.mark.parametrize("NK", [1, 2])
@pytest.mark.parametrize("NB", [5, 6, 8])
def test_no_item_is_overwritten_before_its_readers_are_through(NK, NB):
    G, ring = _constant("kFwdGroups"), _constant("kFwdRing")
    rng = random.Random(NK * 10 + NB)
    streams = [[1] * 40] + [[rng.choice((1, 1, 1, 2, 5)) for _ in range(40)] for _ in range(10)]
    need = {role: max(_published_while(role, held, s, NK, NB, G) for s in streams for held in (8, 9, 10, 11))
            for role in ("group", "loader", "v")}
    assert max(need.values()) <= ring, need


def test_kernel_asserts_the_same_bound():
    assert "static_assert(kFwdRing >= NK + 8" in SOURCE


def test_a_wait_that_runs_out_does_so_for_the_whole_warp():
    """Behind a wait stand shuffles and __syncwarp(): lanes that gave up must not leave the others there."""
    code = re.sub(r"//[^\n]*", "", SOURCE)
    kernel = code[code.index("fwd_main_tc_kernel(TcParams p"):code.index("struct BwdItem")]
    waits = [s for s in re.split(r"[;{}]", kernel) if "mbar_wait(" in s]
    assert len(waits) >= 6
    for s in waits:                               # (the issuer is a single thread)
        assert "__all_sync(0xffffffffu, mbar_wait(" in " ".join(s.split()) or "bar_info" in s or "(np - 1) & 1" in s, s
    # descriptions: the answer is voted on where it is asked for
    asked = [m.end() for m in re.finditer(r"const int total = item_total\(n\);", kernel)]
    assert len(asked) == 3 and kernel.count("item_total(n)") == 3
    for at in asked:
        assert "__all_sync(0xffffffffu, total >= 0);" in kernel[at:at + 80]


@pytest.mark.parametrize("name,kernel,last", [("fmb_attn_tc.cu", "fwd_main_tc_kernel(TcParams p", "bar_fin, (np - 1) & 1"),
                                              ("fmb_gate.cu", "gate_select_kernel(GateParams p", "bar_qfree, (qn - 1) & 1")])
def test_the_last_commit_lands_before_the_cta_ends(name, kernel, last):
    """A commit arrives on a barrier in the CTA's shared memory when its MMAs have completed, whether or not anyone waits for it."""
    code = open(os.path.join(ROOT, "flash_moba_b200", "csrc", name)).read()
    code = code[code.index(kernel):]
    code = code[:code.index("tmem_dealloc(")]
    assert code.rindex("mbar_wait(&" + last) > code.rindex("umma_commit(")
