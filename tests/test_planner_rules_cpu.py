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


def test_direct_cross_products_are_chosen_by_counts_and_lengths(tmp_path):
    """The direct cross-product kernels: the side with more strings gives the texts, few strings on one side or the other
    included; lengths that would leave a warp's threads waiting for its longest text, or a thread on a long chain, stay on
    the planned routes; and no choice lies outside what the kernels take (patterns up to 1,024, 1,536 cells of patterns past
    512)."""
    broken = run_checks(tmp_path, r"""
#include <cstdio>
#include <vector>
#include <cstdlib>
#include "direct_rule.h"
using namespace szs_gb300;
using lengths_t = std::vector<std::uint64_t>;
static direct_extents_t extents(lengths_t const &lengths) {
    direct_extents_t e {};
    for (std::size_t i = 0; i < lengths.size(); ++i) {
        std::uint64_t group = 0;
        for (std::size_t k = i / 32 * 32; k < i / 32 * 32 + 32 && k < lengths.size(); ++k) group = std::max(group, lengths[k]);
        std::uint64_t const n = lengths[i], words = (n + 31) / 32;
        e.longest = std::max(e.longest, n), e.symbols += n, e.padded += group, e.words += words;
        e.words_two += (words + 1) / 2 * 2, e.words_four += (words + 3) / 4 * 4, e.long_words += n > 512 ? words : 0;
    }
    if (lengths.size() % 32) { // the last group's missing strings wait, too
        std::uint64_t group = 0;
        for (std::size_t k = lengths.size() / 32 * 32; k < lengths.size(); ++k) group = std::max(group, lengths[k]);
        e.padded += (32 - lengths.size() % 32) * group;
    }
    return e;
}
static direct_choice_t choose(lengths_t const &q, lengths_t const &c) {
    return direct_choice(extents(q), q.size(), extents(c), c.size());
}
static lengths_t same(std::size_t count, std::uint64_t length) { return lengths_t(count, length); }
static lengths_t mixed(std::size_t count, std::uint64_t low, std::uint64_t high, int one_in) {
    lengths_t lengths(count, low);
    for (std::size_t i = 0; i < count; i += one_in) lengths[i] = high;
    return lengths;
}
static void expect(char const *what, direct_choice_t got, direct_choice_t want) {
    if (got != want) std::printf("%s: %d, not %d\n", what, (int)got, (int)want);
}
int main() {
    expect("1,000,000 x 1 of 150", choose(same(1000000, 150), same(1, 150)), direct_candidates_k);
    expect("1 x 1,000,000 of 150", choose(same(1, 150), same(1000000, 150)), direct_queries_k);
    expect("100,000 x 8 of 150", choose(same(100000, 150), same(8, 150)), direct_candidates_k);
    expect("20,000 x 16 of 800", choose(same(20000, 800), same(16, 800)), direct_candidates_k);
    expect("16 x 20,000 of 800", choose(same(16, 800), same(20000, 800)), direct_queries_k);
    expect("1,000,000 x 1 tokens", choose(same(1000000, 10), same(1, 10)), direct_candidates_k);
    expect("2,048 x 2,048 tokens", choose(same(2048, 10), same(2048, 10)), direct_queries_k);
    expect("197 x 198 of 1,000", choose(same(197, 1000), same(198, 1000)), direct_queries_k);
    expect("2,048 of 8 x 2,048 of 512", choose(same(2048, 8), same(2048, 512)), direct_candidates_k);
    expect("2,048 of 512 x 2,048 of 8", choose(same(2048, 512), same(2048, 8)), direct_queries_k);
    expect("16 x 16 of 150", choose(same(16, 150), same(16, 150)), direct_queries_k);
    expect("a few long ones", choose(mixed(1024, 20, 1000, 33), mixed(1024, 20, 1000, 33)), direct_none_k);
    expect("20,000 of 150 x 40 of 20,000", choose(same(20000, 150), same(40, 20000)), direct_none_k);
    expect("1 of 16 x 1 of 1,000,000", choose(same(1, 16), same(1, 1000000)), direct_none_k);
    expect("40 x 40 of 1,000 x 5,000", choose(same(40, 1000), same(40, 5000)), direct_none_k);
    expect("31 x 31 of 1,000", choose(same(31, 1000), same(31, 1000)), direct_none_k);
    expect("2,000 of 1,025 x 2,000 of 1,025", choose(same(2000, 1025), same(2000, 1025)), direct_none_k);
    expect("2,000 of 1,025 x 2,000 of 100", choose(same(2000, 1025), same(2000, 100)), direct_candidates_k);
    std::srand(1);
    for (int round = 0; round < 3000; ++round) {
        lengths_t sides[2];
        for (auto &side : sides) {
            side.resize(1 + std::rand() % (round % 2 ? 40 : 900));
            int const most = 1 + std::rand() % (round % 3 ? 600 : 2500);
            for (auto &length : side) length = std::rand() % (most + 1);
        }
        direct_choice_t const choice = choose(sides[0], sides[1]);
        if (choice == direct_none_k) continue;
        std::uint64_t const rows = extents(sides[choice == direct_candidates_k]).longest;
        if (rows > 1024 || (rows > 512 && sides[0].size() * sides[1].size() < 1536))
            std::printf("%zu x %zu: patterns of %d\n", sides[0].size(), sides[1].size(), (int)rows);
    }
}
""")
    assert not broken, broken[:5]


def test_small_host_calls_are_chosen_by_their_chains(tmp_path):
    """Few pairs from host memory take the one-kernel path unless a long text beside a short pattern, or many warps, take
    longer there than on the planned routes; the estimate only grows with a call's pairs and lengths."""
    broken = run_checks(tmp_path, r"""
#include <cstdio>
#include "small_rule.h"
using namespace szs_gb300;
static bool pays(int count, std::uint64_t rows, std::uint64_t cols) {
    small_estimate_t estimate;
    for (int i = 0; i < count; ++i) estimate.add(rows, cols);
    return estimate.pays();
}
static void expect(int count, std::uint64_t rows, std::uint64_t cols, bool want) {
    if (pays(count, rows, cols) != want)
        std::printf("%d x (%llu, %llu): not %d\n", count, (unsigned long long)rows, (unsigned long long)cols, (int)want);
}
int main() {
    expect(64, 160, 256, true), expect(1, 1, 1, true), expect(2048, 16, 16, true);
    expect(2048, 200, 200, true), expect(100, 60, 1200, true), expect(64, 200, 5000, true), expect(512, 1000, 1000, true);
    expect(1, 16, 1000000, false), expect(64, 32, 10000, false), expect(4, 100, 200000, false);
    expect(2048, 8, 500, false), expect(2048, 300, 500, false), expect(500, 20, 1500, false);
    for (int rows : {1, 33, 100, 250})
        for (int count : {1, 2048}) {
            bool last = true;
            for (std::uint64_t cols = rows; cols < (1u << 20); cols += 1 + cols / 8) {
                bool const now = pays(count, rows, cols);
                if (now && !last) std::printf("%d x (%d, %d): pays again\n", count, rows, (int)cols);
                last = now;
            }
        }
}
""")
    assert not broken, broken[:5]


def test_quarter_octaves_need_rows(tmp_path):
    """Calls measured faster in halves of octaves stay there, and those measured faster in quarters have rows enough."""
    broken = run_checks(tmp_path, r"""
#include <cuda_runtime.h>
#include <cstdio>
#include "planner.cuh"
using namespace szs_gb300;
static void expect(double pairs, float rows, float columns, bool profile, bool want) {
    if ((pairs * rows >= short_fine_rows(rows, columns, profile)) != want)
        std::printf("%.0f pairs of %.0f x %.0f, profile %d: not %d\n", pairs, rows, columns, (int)profile, (int)want);
}
int main() {
    expect(150000, 30, 600, true, false), expect(45000, 30, 600, false, false), expect(250000, 30, 600, false, true);
    expect(20000, 167, 233, true, false), expect(45000, 167, 233, true, true), expect(30000, 167, 233, false, true);
    expect(65536, 93, 147, true, false), expect(100000, 93, 147, true, true), expect(65536, 93, 147, false, true);
    expect(20000, 200, 200, true, false), expect(65536, 200, 200, true, true), expect(65536, 200, 200, false, true);
    expect(65536, 120, 120, true, true), expect(1048576, 72, 72, true, true), expect(16384, 350, 350, true, true);
    expect(150000, 53, 91, true, false), expect(150000, 53, 91, false, true), expect(16384, 450, 450, false, true);
}
""")
    assert not broken, broken[:5]


def test_near_diagonal_trials_that_pay(tmp_path):
    """The trial near the diagonal: small calls need hardly an unrelated pair and their longest pairs well inside the
    limit, large ones enough alike; calls measured faster without it go without."""
    broken = run_checks(tmp_path, r"""
#include <cuda_runtime.h>
#include <cstdio>
#include "planner.cuh"
using namespace szs_gb300;
static void expect(char const *what, double unrelated, double alike, double rate, std::uint64_t pairs, unsigned longest,
                   int half, bool want) {
    near_sample_t const sample {128, unsigned(128 * unrelated), unsigned(128 * alike),
                                unsigned((128 - unsigned(128 * unrelated)) * 32 * rate)};
    if (near_pays(sample, pairs, longest, half) != want) std::printf("%s: not %d\n", what, (int)want);
}
int main() {
    expect("1M reads, 4 %", 0, 1, 0.04, 1 << 20, 300, 1, true), expect("long reads, 4 %", 0, 1, 0.04, 4096, 4000, 4, true);
    expect("65,536 CJK, 7 %", 0, 1, 0.07, 65536, 300, 1, true), expect("20,000 reads, 10 %", 0, 1, 0.10, 20000, 300, 1, true);
    expect("20,000 reads, 17 %", 0, 0.9, 0.17, 20000, 300, 1, false);
    expect("20,000 reads, a tenth unrelated", 0.1, 0.9, 0.02, 20000, 300, 1, false);
    expect("200,000 reads, a third unrelated", 0.35, 0.65, 0.02, 200000, 300, 1, true);
    expect("200,000 reads, two thirds unrelated", 0.65, 0.35, 0.02, 200000, 300, 1, false);
    expect("5,000 long reads, a tenth unrelated", 0.1, 0.9, 0.02, 5000, 4000, 4, false);
    expect("5,000 long reads, 9 %", 0, 0.2, 0.09, 5000, 4000, 4, false);
    expect("unrelated", 1, 0, 0, 1 << 20, 300, 1, false), expect("20,000 unrelated", 1, 0, 0, 20000, 300, 1, false);
    near_sample_t const none {};
    if (near_pays(none, 1 << 20, 300, 1) || near_pays(none, 1000, 300, 1)) std::printf("nothing sampled\n");
}
""")
    assert not broken, broken[:5]
