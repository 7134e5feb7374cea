"""What PTX asks of a thread that issues MMAs, by the text of the sources: behind a wait for a barrier by which other warps say that they have read or
written Tensor Memory, and ahead of the MMA that relies on it, stands tcgen05.fence::after_thread_sync."""
import re

import pytest

from test_follow_on_cpu import KERNELS

# a wait: one of the bounded waits (or the issuers' shorthand for it), or a test that lets the thread go on
STEP = re.compile(r"\b(?:(?P<wait>mbar_wait|mbar_spin|mbar_test|wait|wait_all)\(&|(?P<fence>tc_fence_after_sync)\(\)|(?P<mma>umma_gemm)<)")
ISSUERS = sorted(n for n, (_, body) in KERNELS.items() if "umma_gemm<" in body)


def test_the_issuers_are_found():
    assert {"fwd_main_tc_kernel", "bwd_main_tc_kernel", "fwd_wide_tc_kernel", "bwd_wide_tc_kernel", "gate_select_kernel"} <= set(ISSUERS)


@pytest.mark.parametrize("name", ISSUERS)
def test_a_fence_between_every_wait_and_the_next_mma(name):
    body, open_wait = KERNELS[name][1], None
    for m in STEP.finditer(body):
        if m["wait"]:
            open_wait = body[m.start():body.index("\n", m.start())]
        elif m["fence"]:
            open_wait = None
        else:
            assert open_wait is None, f"no fence between '{open_wait}' and '{body[m.start():body.index(';', m.start())]}'"
