"""runs.hpp (host code): the room for experts' results covers every step of up to R rows, is not larger than that, and takes a moment to work out."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "fastllm_b200" / "csrc"
PROGRAM = r"""
#include "runs.hpp"
#include <chrono>
#include <cstdio>
int main() {
    for (int top : {1, 2, 3, 8})
        for (int experts : {1, 2, 8, 37, 300})
            for (int ff : {512, 2816, 14336})
                for (int R : {128, 129, 130, 257, 700, 3000}) {
                    if (top > experts) continue;
                    size_t want = 0;
                    for (int T = 129; T <= R; ++T) {
                        const int ks = fl::runs_ksplit(T * top, experts, 2048, ff, 148), nk = (ff + 63) / 64;
                        if (ks < 1 || ks > 4 || (ks > 1 && (nk + ks - 1) / ks * (ks - 1) >= nk)) return 1;
                        want = std::max(want, ks * fl::run_capacity(T * top, experts));
                    }
                    if (fl::runs_most_rows(top, experts, 2048, ff, 148, R) != want) { std::printf("%d %d %d %d\n", top, experts, ff, R); return 2; }
                }
    const auto t0 = std::chrono::steady_clock::now();
    volatile size_t rows = fl::runs_most_rows(2, 8, 4096, 14336, 148, 1 << 20);
    (void)rows;
    return std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count() < 0.02 ? 0 : 3;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_room_for_the_results_of_every_step(tmp_path):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", str(CSRC), "-o", str(tmp_path / "t"), str(tmp_path / "t.cpp")], check=True)
    assert subprocess.run([str(tmp_path / "t")], timeout=120).returncode == 0
