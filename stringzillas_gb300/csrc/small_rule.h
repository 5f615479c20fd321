/**
 *  @file small_rule.h
 *  @brief Which small pairwise calls from host memory take the one-kernel path (small.cu) instead of the planned routes.
 *
 *  The one-kernel path saves some 80 us of planning, launches and copies per call, and then scores a pair on a warp at one
 *  word per lane: a column takes a step however few words the pattern has. The planned thread-per-pair kernels take a
 *  column of a one-word pattern in a quarter of that time, so texts of more than about a thousand symbols beside short
 *  patterns belong there, and so do large calls whose warps wait for issue slots. Both are estimated in nanoseconds, as the
 *  larger of the longest pair's chain and all pairs' steps. Fitted to whole calls on a GB300 (one kernel / planned): 64
 *  pairs of 32 x 10,000 867 / 413 us, one of 16 x 1,000,000 78.5 / 20.5 ms, 2,048 of 300 x 500 250 / 203 us, 500 of 20 x
 *  1,500 203 / 179, which are now planned; 64 of 200 x 5,000 459 / 585, 2,048 of 200 x 200 122 / 157, 100 of 60 x 1,200
 *  145 / 159, 512 of 1,000 x 1,000 195 / 305, which are not.
 */
#pragma once
#include <algorithm>
#include <cstdint>

namespace szs_gb300 {

/** In nanoseconds and picoseconds: whole numbers, since the host adds up every pair of a call before it does anything. */
struct small_estimate_t {
    std::uint64_t chain_ns = 0, steps_ps = 0;                 // one kernel: the longest pair, all of them
    std::uint64_t planned_chain_ns = 0, planned_steps_ps = 0; // planned routes

    /** A pair of `rows` (at most 1,024) and `cols` symbols. */
    void add(std::uint64_t rows, std::uint64_t cols) {
        std::uint64_t const words = (rows + 31) / 32, columns = cols + words;
        bool const tabled = rows <= 256, thread = rows <= 512; // match masks in shared memory; a thread per pair if planned
        chain_ns = std::max(chain_ns, columns * (tabled ? 79 : 87));
        steps_ps += columns * (tabled ? 117 : 185);
        planned_chain_ns = std::max(planned_chain_ns, cols * (thread ? 9 + 11 * words : 80));
        planned_steps_ps += thread ? 0 : columns * 170;
    }
    bool pays() const {
        return 48000 + std::max(chain_ns, steps_ps / 1000) < 130000 + std::max(planned_chain_ns, planned_steps_ps / 1000);
    }
};

} // namespace szs_gb300
