"""The tcgen05 attention kernels' softmax threads may touch the accumulator only behind the P.V products it still has to take.  An mbarrier
wait names a parity, not a phase, so each wait has to hold for EVERY number of products that can be complete when it is reached: the waits
are read out of the kernels' source and run against a model of the barriers."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "fastllm_b200" / "csrc"


def waits(path, kernel, pages):
    """[(barrier, index, parity)] as Python expressions of j, b and the page count: rescale, reuse of the P buffer, end"""
    body = path.read_text().split(kernel, 1)[1].split("tcgen05.dealloc", 1)[0]
    found = re.findall(r"(?:mbar_wait|gt_wait)\(&(o_done|p_free)(?:\[([^\]]*)\])?, ([^;]*?)\)\)?;", body)
    assert len(found) == 3, found
    return [(n, (i or "0").replace(pages, "np"), p.replace(pages, "np")) for n, i, p in found]


@pytest.mark.parametrize("name,kernel,pages", [("gqa_attn_tc.cuh", "ly_gqa_tc_kernel(", "np"), ("attn_mma.cuh", "attn_prefill_tc_kernel(", "nkt")])
@pytest.mark.parametrize("np", [1, 2, 3, 4, 5, 9, 64])
def test_waits_name_one_phase(name, kernel, pages, np):
    rescale, reuse, end = waits(CSRC / name, kernel, pages)
    known = 0                                   # products that earlier waits have shown to be complete

    def passes(wait, j, complete):              # `complete` products are over: has the barrier left the phase of this parity?
        barrier, index, parity = wait
        env = {"j": j, "b": j & 1, "np": np}
        at, par = eval(index, {}, env), eval(parity, {}, env)
        phases = complete if barrier == "o_done" else sum(1 for i in range(complete) if i & 1 == at)
        return phases & 1 != par

    def check(wait, j, need, most):
        for c in range(known, most + 1):
            assert passes(wait, j, c) == (c >= need), f"page {j} of {np}: {c} products complete, {need} needed"

    for j in range(np):
        if j > 0:
            check(rescale, j, j, j)             # (whether a row's maximum moves is up to the data: nothing is known from this one)
        check(reuse, j, max(0, j - 1), j)
        known = max(known, j - 1)
    check(end, np, np, np)
