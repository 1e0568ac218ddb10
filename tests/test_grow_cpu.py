"""grow.hpp (host code): a size counts as had only when every buffer of it is there."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "fastllm_b200" / "csrc"
PROGRAM = r"""
#include "grow.hpp"
#include <stdexcept>
int main() {
    size_t cap = 0, first = 0, second = 0;
    int calls = 0;
    bool fail = false;
    auto call = [&](size_t want) {
        fl::grow(cap, want, [&] {
            ++calls;
            first = want; second = 0;
            if (fail) throw std::runtime_error("no memory");
            second = want;
        });
        return cap >= want && first >= want && second >= want;
    };
    if (!call(10) || !call(7) || calls != 1) return 1;          // smaller calls take nothing
    fail = true;
    for (int i = 0; i < 2; ++i) {                               // the same call again: it may not go on without its second buffer
        try { call(20); return 2; } catch (const std::runtime_error&) {}
        if (cap != 0) return 3;
    }
    fail = false;
    if (!call(7) || !call(20) || calls != 5) return 4;          // what was had before is gone too
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_sizes_count_once_the_buffers_are_there(tmp_path):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CSRC}", str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    assert subprocess.run([str(tmp_path / "t")]).returncode == 0


def test_the_encoder_reserves_through_it():
    body = (CSRC / "fl_bert.cu").read_text().split("static void bert_reserve(", 1)[1].split("\n}\n", 1)[0]
    for cap in ("cap_chain", "cap_tokens", "cap_batch"):
        assert f"grow(m.{cap}, " in body and f"m.{cap} =" not in body


def test_one_decision_for_buffers_and_launches():
    """bert_run alone asks which kernels take a call: reserving and launching on answers of their own could differ"""
    source = (CSRC / "fl_bert.cu").read_text()
    calls = source.count("bert_blocks(m,")
    assert calls == 1 and "bert_blocks(m, b * t)" in source.split("static BertRun bert_run(", 1)[1].split("\n}\n", 1)[0]


def test_nothing_is_taken_between_a_step_and_its_logits():
    """a step that has run has moved the cache on: memory for its delivery that cannot be had then would cost the cache, and page-locking takes
    milliseconds of the call"""
    source = (CSRC / "fl_lib.cu").read_text()
    deliver = source.split("static void logits_to_host(", 1)[1].split("\n}\n", 1)[0]
    sample = source.split("FL_EXPORT int fl_forward_sample(", 1)[1].split("FL_API_END", 1)[0]
    assert ".alloc(" not in deliver and ".alloc(" not in sample
    assert "c.h_logits.alloc(" in source.split("static void cache_create(", 1)[1].split("\n}\n", 1)[0]
    assert "y.h_logits.alloc(" in (CSRC / "fl_layered.cu").read_text().split("static void ensure_ws(", 1)[1].split("\n}\n", 1)[0]


def test_repeats_ask_for_every_buffer():
    """an embedding in another thread may have failed to grow the workspace in between: a repeat looks at all three sizes"""
    body = (CSRC / "fl_bert.cu").read_text().split("void bert_repeat(", 1)[1].split("\n}\n", 1)[0]
    assert all(f"<= m.{cap}" in body for cap in ("cap_tokens", "cap_batch", "cap_chain"))
