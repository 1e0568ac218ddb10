"""Kernels on pairs of SMs: a wait that acquires at cluster scope pairs only with arrives that release there (PTX: without a scope an
arrive is ordered within its CTA alone), so no arrive on the other CTA's barrier may leave the scope out.  Read out of the sources."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "fastllm_b200" / "csrc"


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cu*")), ids=lambda p: p.name)
def test_remote_arrives_release_at_cluster_scope(path):
    remote = re.findall(r"mbarrier\.arrive[\w.:]*\.shared::cluster[\w.:]*", path.read_text())
    assert all(".release.cluster." in a for a in remote), remote
    if path.name == "gemm_pair.cuh":
        assert remote
