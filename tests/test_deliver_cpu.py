"""deliver_logits (host code) over a fake device: the caller's buffer holds the logits behind a good step and is untouched behind a failed one."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "fastllm_b200" / "csrc"
PROGRAM = r"""
#include "deliver.hpp"
#include <cstdio>
#include <stdexcept>
#include <vector>
// fail: 0 never, 1 the step's kernels (the first wait), 2 a peer that was missed (the check)
struct Fake {
    std::vector<float>& pinned; int fail; size_t end = 0; int parts = 0, fetched = 0, waited = 0, checked = 0;
    void begin(int n) { parts = n; }
    void fetch(int p, size_t at, size_t count) { if (p != fetched++ || at != end) throw std::logic_error("parts out of order"); end = at + count; }
    void wait(int p) {
        if (p != waited++) throw std::logic_error("waits out of order");
        if (fail == 1) throw std::runtime_error("step");
        for (size_t i = 0; i < pinned.size(); ++i) pinned[i] = (float)i;
    }
    void check() { ++checked; if (waited != 1) throw std::logic_error("checked late"); if (fail == 2) throw std::runtime_error("peer"); }
};
int main() {
    const size_t line = 1024 * 1024;      // floats: two parts from here on
    for (size_t n : {(size_t)1, (size_t)31999, line - 1, line, line + 1, 5 * line / 2 + 3, 20 * line})
        for (int fail = 0; fail < 3; ++fail) {
            std::vector<float> pinned(n), host(n, -1.f);
            Fake f{pinned, fail};
            bool threw = false;
            try { fl::deliver_logits(f, pinned.data(), host.data(), n); } catch (const std::runtime_error&) { threw = true; }
            if (threw != (fail != 0) || f.end != n || f.fetched != f.parts || (f.parts > 1) != (n >= line)) return std::printf("n %zu fail %d\n", n, fail), 1;
            for (size_t i = 0; i < n; ++i)
                if (host[i] != (fail ? -1.f : (float)i)) return std::printf("n %zu fail %d: %zu\n", n, fail, i), 1;
        }
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_buffer_behind_good_and_failed_steps(tmp_path):
    src, exe = tmp_path / "deliver.cpp", tmp_path / "deliver"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
