"""Kernels on pairs of SMs: a wait that acquires at cluster scope pairs only with arrives that release there (PTX: without a scope an
arrive is ordered within its CTA alone), so no arrive on the other CTA's barrier may leave the scope out, and what hands over memory releases.
Read out of the sources."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "fastllm_b200" / "csrc"


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cu*")), ids=lambda p: p.name)
def test_remote_arrives_release_at_cluster_scope(path):
    remote = re.findall(r"mbarrier\.arrive[\w.:]*\.shared::cluster[\w.:]*", path.read_text())
    assert all(".release.cluster." in a or ".relaxed.cluster." in a for a in remote), remote
    if path.name == "gemm_pair.cuh":
        assert remote


def test_relaxed_arrives_hand_over_no_memory():
    """the encoder block's operands (x_ready, h_ready) go through `arrive`, which releases; only S, which lies in registers by then, may do without"""
    body = (CSRC / "bert_block.cuh").read_text()
    assert re.findall(r"mbar_arrive_cluster_relaxed\(mapa_u32\(smem_u32\(&(\w+)\)", body) == ["s_free"]
    assert sorted(re.findall(r" arrive\(&(\w+)\);", body)) == ["h_ready", "x_ready"]
    assert "mbar_arrive_cluster_relaxed(m" not in (CSRC / "gemm_pair.cuh").read_text()
