"""Kernels that bring operands with bulk copies and give up on a wait that runs out: what such a block still has in flight has to land before it ends, and
the host has to hear of it.  Read out of the sources."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "fastllm_b200" / "csrc"


@pytest.mark.parametrize("path,name", [("bert_small.cuh", ") bert_small_kernel"), ("bert_qkv.cuh", "\nbert_qkv_attn_kernel"), ("bert_block.cuh", "\nbert_block_kernel"),
                                       ("layered_ops.cuh", ") ly_rec_scan_kernel")])
def test_a_wait_that_runs_out(path, name):
    body = (CSRC / path).read_text().split(f"{name}(", 1)[1].split("\n}\n", 1)[0]
    assert re.search(r"\bmbar_wait\(", body) is None, "a wait without a limit"
    assert re.search(r"\b(pair_wait|mbar_wait_bounded)\(", body)
    end = re.search(r"failed != nullptr\) \*\w+\.failed = 1;\s*for \(int i = 0; i < 1000; \+\+i\) __nanosleep\(1000\);", body)
    assert end, "a block that gave up reports it and waits for its copies"
