"""Kernels that are brought up while the kernel before them on the stream still runs, by the text of the sources: each waits for
that kernel before anything else, and none reads global memory in a way that counts on data that nobody writes while the
kernel exists (ld.global.nc, and what the compiler may make of a const __restrict__ parameter)."""
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "flash_moba_b200", "csrc")


def _code(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


def _block(text, at):
    """The brace block that opens at or behind `at`."""
    start = at = text.index("{", at)
    depth = 0
    while True:
        depth += {"{": 1, "}": -1}.get(text[at], 0)
        at += 1
        if depth == 0:
            return text[start + 1:at - 1]


FILES = {f: _code(f) for f in sorted(os.listdir(CSRC)) if f.endswith((".cu", ".cuh"))}
KERNELS = {}      # name -> (parameters, body)
for _t in FILES.values():
    for _m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\(", _t):
        KERNELS[_m.group(1)] = (_t[_m.end():_t.index("{", _m.end())], _block(_t, _m.end()))


def _launched_early():
    names = set()
    for text in FILES.values():
        starts = [m.end() for m in re.finditer(r"launch_follow_on\(", text)]
        starts += [m.start() for m in re.finditer(r"cudaLaunchKernelEx\(&cfg, ", text)]
        for at in starts:
            what = re.match(r"(?:cudaLaunchKernelEx\(&cfg, )?(\w+)", text[at:]).group(1)
            if what in KERNELS:
                names.add(what)
                continue
            made = [m for m in re.finditer(r"auto %s = ([^;]*);" % what, text[:at])]      # (the helper itself has a parameter instead)
            names |= {w for w in re.findall(r"\w+", made[-1].group(1)) if w in KERNELS} if made else set()
    return names


EARLY = _launched_early()


def _readers_of_constant_data():
    """Device functions that use non-coherent loads, directly or through others."""
    found = {m.group(1) for t in FILES.values() for m in re.finditer(r"__forceinline__ [\w:<>&*]+ (\w+)\([^)]*\) \{", t)
             if "ld.global.nc" in _block(t, m.end() - 1)}
    assert found                                   # ordinary kernels do use such a load
    while True:
        more = {m.group(1) for t in FILES.values() for m in re.finditer(r"(?:__forceinline__|static __device__) \S+ (\w+)\(", t)
                if any(re.search(r"\b%s\b" % f, _block(t, m.end())) for f in found)}
        if more <= found:
            return found
        found |= more


def test_the_kernels_are_found():
    assert {"dot_do_o_kernel", "decode_kernel", "fwd_main_tc_kernel", "bwd_main_tc_kernel", "fwd_wide_tc_kernel", "bwd_wide_tc_kernel",
            "gate_select_kernel", "csc_tile_hist_kernel", "csc_tile_scan_kernel", "csc_scatter_kernel"} <= EARLY
    assert not {"merge_kernel", "mean_pool_kernel"} & EARLY


@pytest.mark.parametrize("name", sorted(EARLY))
def test_waits_first_and_reads_coherently(name):
    params, body = KERNELS[name]
    before, found, _ = body.partition("follow_on();")
    assert found
    for statement in before.split(";"):
        assert re.match(r"\s*(constexpr\b|using\b|static_assert\b|$)", statement), statement
    assert "__restrict__" not in params
    assert "__ldg" not in body and "ld.global.nc" not in body
    used = [f for f in _readers_of_constant_data() if re.search(r"\b%s\b" % f, body)]
    assert not used, used
