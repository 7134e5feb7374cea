"""The candidate queues of the two-sweep gating kernel against their room: the rules by which a thread's queue grows and is cut, with the
kernel's own constants, over streams in which every score, or whole runs of scores, reach the floor.  (A queue that outgrows its room
writes into another row's: lists that are wrong now and then, and only in row tiles with rows of several warps.)"""
import os
import random
import re

import pytest

from conftest import ROOT

SOURCE = open(os.path.join(ROOT, "flash_moba_b200", "csrc", "fmb_gate.cu")).read()


def _pick(pattern, kmax):
    """The constant that `KMAX == 8 ? a : b` names."""
    m = re.search(pattern + r"[^;]*KMAX == 8 \? (\d+) : (\d+);", SOURCE)
    return int(m.group(1 if kmax == 8 else 2))


def _longest(streams, cap, step, need, one_by_one):
    """Most entries of any queue of a warp's threads; `streams`: per thread, which of its scores reach the floor."""
    cnt, most = [0] * len(streams), 0
    for at in range(0, len(streams[0]), step):
        near_full = any(c > cap - step for c in cnt)
        if near_full and not one_by_one:
            cnt = [min(c, need) for c in cnt]
        for j in range(at, at + step):
            if near_full and one_by_one and any(c == cap for c in cnt):
                cnt = [min(c, need) for c in cnt]
            cnt = [c + s[j] for c, s in zip(cnt, streams)]
            most = max(most, *cnt)
    return most


@pytest.mark.parametrize("kmax", [8, 16])
def test_no_queue_outgrows_its_room(kmax):
    cap, step = _pick(r"sel_cap\(\)", kmax), _pick(r"(?:sel_step\(\)|constexpr int STEP)", kmax)
    one_by_one = kmax + step > cap and "sel_append4(queue, cnt, CAP, need" in SOURCE
    rng = random.Random(kmax)
    for need in range(0, kmax + 1):
        for density in (1.0, 0.97, 0.8, 0.5):
            streams = [[1 if rng.random() < density else 0 for _ in range(512)] for _ in range(4)]
            streams[0] = [1] * 512 if density == 1.0 else streams[0]
            for quiet in (0, 3, 15, 16, 17):         # a run of candidates, then none, then a run again
                cut = [s[:quiet] + [0] * (-quiet % step) + s[quiet:] for s in streams]
                cut = [s[:len(s) // step * step] for s in cut]
                assert _longest(cut, cap, step, need, one_by_one) <= cap, (need, density, quiet)


def test_every_cta_writes_its_lists():
    """The lists' memory is not initialised, and the status word is read on request only: a CTA that leaves before it has written
    its lists would hand what the memory held before to the pattern builder."""
    code = re.sub(r"//[^\n]*", "", SOURCE[SOURCE.index("\ngate_select_kernel(GateParams p"):])
    code = code[:code.index("tmem_dealloc(")]
    assert re.findall(r"\breturn\b *;", code) == []
