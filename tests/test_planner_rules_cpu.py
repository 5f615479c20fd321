"""The planner's host-callable rules, compiled from their header with the host compiler and checked over their whole
ranges: no GPU."""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "stringzillas_gb300", "csrc")


def run_checks(tmp_path, source):
    """Builds a program that includes the engine's headers and prints one line per broken rule; returns its lines."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    compiler = shutil.which("g++")
    if not compiler or not os.path.exists(nvcc):
        pytest.skip("needs g++ and the CUDA headers")
    (tmp_path / "checks.cpp").write_text(source)
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    subprocess.run([compiler, "-std=c++17", "-O1", "-I", include, "-I", os.path.join(REPO, "include"), "-I", CSRC,
                    str(tmp_path / "checks.cpp"), "-o", str(tmp_path / "checks")], check=True, capture_output=True)
    return subprocess.run([str(tmp_path / "checks")], check=True, capture_output=True, text=True).stdout.splitlines()


def test_short_bins_hold_every_text_length(tmp_path):
    """Every short pair's bin lies in its shape's range, whatever its text's length (a local pair's may pass 2^31), and
    longer texts never come in later bins of it."""
    broken = run_checks(tmp_path, r"""
#include <cuda_runtime.h>
#include <cstdio>
#include "planner.cuh"
using namespace szs_gb300;
int main() {
    for (int fine = 0; fine < 2; ++fine)
        for (std::uint64_t n = 1; n <= short_max_rows_k; ++n) {
            int shape = 0;
            while (short_segment_rows(shape) < (int)n || (!fine && shape % 2)) ++shape;
            int const begin = bin_short_begin_k + shape * short_m_classes_k, end = begin + short_m_classes_k;
            int last = end;
            for (std::uint64_t m = n, step = 1; m < (1ull << 32); m += step, step += m / 64 > step ? step : 0) {
                int const key = short_bin(n, m, fine != 0);
                if (key < begin || key >= end || key > last) {
                    std::printf("n %d m %llu: bin %d of [%d, %d), after %d\n", (int)n, (unsigned long long)m, key, begin,
                                end, last);
                    break;
                }
                last = key;
            }
            int const longest = short_bin(n, 0xFFFFFFFFull, fine != 0);
            if (longest != begin) std::printf("n %d, the longest text: bin %d, not %d\n", (int)n, longest, begin);
        }
}
""")
    assert not broken, broken[:5]
