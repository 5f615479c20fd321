/**
 *  @file myers_warp.cuh
 *  @brief Unit-cost Levenshtein by the bit-parallel method for patterns of 513 to 8,192 characters: one warp per
 *         pair, the pattern's words spread over the lanes, the text swept through the lanes as a pipeline.
 *
 *  The thread-per-pair kernel (myers.cuh) keeps a whole pattern of up to 16 words in one thread's registers. A longer
 *  pattern is cut into 32 slices of W words (W = ceil(n / 1,024) <= 8): lane L holds rows [32 W L, 32 W (L + 1)).
 *  One column of the bit-parallel step needs, for lane L's lowest word, three bits of lane L - 1's highest word in
 *  the same column: the carry out of the multi-word add and the top bits of the horizontal deltas Ph and Mh that are
 *  shifted in. So at step t lane L scores text column t - L, and lane L + 1 takes the carry and the two delta bits
 *  from lane L one step later in one shuffle; the column's character travels a step ahead in another. Lane 0 shifts +1
 *  into row 0 (the top row grows by one per column) and nothing into the carry; it takes the text from chunks of 32
 *  characters that the warp loads together a chunk ahead. Nothing keeps the score per column: after the last one the
 *  vertical deltas of rows 1..n, summed over the lanes, lead from the top row's D[0][m] = m to the distance. The steps
 *  in which every lane is inside the text take no range checks. A step is one warp's chain of dependent instructions, so
 *  what it waits for decides, at few pairs and at many: with the symbol in the same shuffle as the bits (its selectors
 *  looked up inside the chain) and the score kept per column, 4,096 unrelated DNA pairs of 1,000-4,000 took 2.04 ms, now
 *  1.35; 55 pairs of 2,351-4,791 1.35 ms, now 0.92; one pair of 8,000 2.41 ms, now 1.31.
 *
 *  The reference reaches patterns of 2,048 characters with its Myers tiers (include/stringzillas/similarities/
 *  cuda.cuh:2072-2634); its serial engine (serial.hpp:1656-1865) answers unit-cost Levenshtein exactly the same way.
 */
#pragma once
#include "myers.cuh"

namespace szs_gb300 {

/** The distance of one pair, computed by the whole warp; every lane returns it. `wide_`: strings of 16-bit codes
 *  (their own codes, selectors from the code's bits), else bytes mapped through the batch alphabet. */
template <int words_, int bits_, bool wide_ = false>
__device__ __forceinline__ std::uint32_t myers_warp_distance(pair_task_t const &task, std::uint8_t const *code,
                                                             plane_selectors_t<bits_> const *selectors) {
    constexpr int W = words_, B = bits_;
    int const lane = threadIdx.x & 31;
    std::uint32_t const n = task.rows_length, m = task.cols_length;
    int const lanes_used = int((n + 32u * W - 1) / (32u * W));

    // This lane's slice of the pattern as B bit planes of its characters' codes.
    std::uint32_t planes[B][W];
    std::uint32_t const lane_base = (std::uint32_t)lane * 32u * W;
#pragma unroll
    for (int w = 0; w < W; ++w) {
        std::uint32_t acc[B];
#pragma unroll
        for (int b = 0; b < B; ++b) acc[b] = 0;
        std::uint32_t const base = lane_base + 32u * w;
        std::uint32_t const valid = n > base ? min(32u, n - base) : 0u;
        for (std::uint32_t k = 0; k < valid; ++k) {
            std::uint32_t const c = wide_ ? symbol_at<true>(task.rows, base + k) : code[task.rows[base + k]];
#pragma unroll
            for (int b = 0; b < B; ++b) acc[b] |= ((c >> b) & 1u) << k;
        }
#pragma unroll
        for (int b = 0; b < B; ++b) planes[b][w] = acc[b];
    }
    std::uint32_t pv[W], mv[W];
#pragma unroll
    for (int w = 0; w < W; ++w) pv[w] = 0xFFFFFFFFu, mv[w] = 0u;

    // Match mask of this lane's rows with one symbol. Its selectors come from shared memory, but where a step is short (one
    // word per lane) those of 8 planes, two 16-byte loads from scattered rows, keep the banks busy longer than the step
    // itself: they are made from the bits of the code, which travels in the symbol's place (60,000 text pairs of 700-1,000
    // 5.5 -> 4.6 ms, 30,000 of 520-700 2.06 -> 1.76; with two to four words per lane the loads are the faster way, 5,000 of
    // 1,000-4,000 2.26 against 2.50).
    constexpr bool codes = wide_ || (B >= 8 && W == 1);
    auto matches = [&](std::uint32_t symbol, std::uint32_t (&eq)[W]) {
        std::uint32_t select[B];
        if constexpr (codes) code_selectors<B>(symbol, select);
        else {
#pragma unroll
            for (int b = 0; b < B; ++b) select[b] = selectors->select[symbol][b];
        }
#pragma unroll
        for (int w = 0; w < W; ++w) {
            eq[w] = 0xFFFFFFFFu;
#pragma unroll
            for (int b = 0; b < B; ++b) eq[w] &= planes[b][w] ^ select[b];
        }
    };
    auto text = [&](std::uint32_t j) -> std::uint32_t {
        std::uint32_t const symbol = j < m ? symbol_at<wide_>(task.cols, j) : 0u;
        return codes && !wide_ ? code[symbol] : symbol;
    };
    std::uint32_t chunk = text(lane), chunk_ahead = text(32u + lane); // columns (t + 1 & ~31) + lane, and 32 later
    std::uint32_t symbol = lane == 0 ? chunk : 0u;
    std::uint32_t eq[W];
    matches(symbol, eq);
    std::uint32_t out = 0; // to lane + 1: carry | top Ph bit << 1 | top Mh bit << 2
    std::uint32_t const steps = m + (std::uint32_t)lanes_used - 1;
    // One step; `inside`: every lane that holds rows is on a column of the text, and the others may compute filler. The
    // symbol travels a step ahead of the three bits, so its match masks are ready when these arrive.
    auto step = [&](std::uint32_t t, bool inside) {
        std::uint32_t in = __shfl_up_sync(0xFFFFFFFFu, out, 1);
        if (lane == 0) in = 2u; // no carry into row 0; +1 shifted into its horizontal delta
        if (((t + 1) & 31u) == 0) chunk = chunk_ahead, chunk_ahead = text(t + 33u + lane);
        std::uint32_t const staged = __shfl_sync(0xFFFFFFFFu, chunk, int((t + 1) & 31u));
        std::uint32_t symbol_next = __shfl_up_sync(0xFFFFFFFFu, symbol, 1);
        if (lane == 0) symbol_next = staged;
        std::uint32_t eq_next[W];
        matches(symbol_next, eq_next);
        int const j = (int)t - lane;
        if (inside || (lane < lanes_used && j >= 0 && j < (int)m)) {
            std::uint32_t xv[W], sum[W];
#pragma unroll
            for (int w = 0; w < W; ++w) xv[w] = eq[w] | mv[w], sum[w] = eq[w] & pv[w];
            // Multi-word (Eq & Pv) + Pv with the carry from the lane below: the carry flag starts as that bit.
            std::uint32_t const carry_in = in & 1u;
            std::uint32_t carry_out, scratch;
            asm volatile("add.cc.u32 %0, %1, 0xFFFFFFFF;" : "=r"(scratch) : "r"(carry_in));
#pragma unroll
            for (int w = 0; w < W; ++w) asm volatile("addc.cc.u32 %0, %0, %1;" : "+r"(sum[w]) : "r"(pv[w]));
            asm volatile("addc.u32 %0, 0, 0;" : "=r"(carry_out));
            std::uint32_t ph_prev = in << 30, mh_prev = in << 29; // their top bits count
#pragma unroll
            for (int w = 0; w < W; ++w) {
                std::uint32_t const xh = (sum[w] ^ pv[w]) | eq[w];
                std::uint32_t const ph = mv[w] | ~(xh | pv[w]);
                std::uint32_t const mh = pv[w] & xh;
                std::uint32_t const ph_shifted = __funnelshift_l(ph_prev, ph, 1);
                std::uint32_t const mh_shifted = __funnelshift_l(mh_prev, mh, 1);
                pv[w] = mh_shifted | ~(xv[w] | ph_shifted);
                mv[w] = ph_shifted & xv[w];
                ph_prev = ph, mh_prev = mh;
            }
            out = carry_out | (ph_prev >> 31) << 1 | (mh_prev >> 31) << 2;
        }
        symbol = symbol_next;
#pragma unroll
        for (int w = 0; w < W; ++w) eq[w] = eq_next[w];
    };
    std::uint32_t const fill = min(steps, (std::uint32_t)lanes_used - 1);
    std::uint32_t t = 0;
    for (; t < fill; ++t) step(t, false);
    for (; t < m; ++t) step(t, true);
    for (; t < steps; ++t) step(t, false);

    // After the last column the vertical deltas of rows 1..n lead from the top row's D[0][m] = m to the distance.
    std::int32_t delta = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
        std::uint32_t const base = lane_base + 32u * w;
        std::uint32_t const rows = n > base ? min(32u, n - base) : 0u;
        std::uint32_t const mask = rows == 32u ? 0xFFFFFFFFu : (1u << rows) - 1u;
        delta += __popc(pv[w] & mask) - __popc(mv[w] & mask);
    }
    return m + (std::uint32_t)__reduce_add_sync(0xFFFFFFFFu, delta);
}

/** Warp-per-pair kernel over bins [key_begin, key_end) with at most `words_` words per lane; warps pull pairs from
 *  the first bin's cursor. With `list` (pairs the near-diagonal kernel left), over the listed tasks of its words. */
template <int words_, int bits_>
__global__ void __launch_bounds__(256) myers_warp_kernel(pair_task_t const *__restrict__ tasks,
                                                         plan_bins_t *__restrict__ bins, int key_begin, int key_end,
                                                         batch_alphabet_t const *__restrict__ alphabet,
                                                         std::int64_t *__restrict__ results,
                                                         std::uint32_t const *__restrict__ list) {
    __shared__ std::uint8_t code_s[256];
    __shared__ plane_selectors_t<bits_> selectors_s;
    for (int i = threadIdx.x; i < 256; i += blockDim.x) {
        std::uint32_t const c = alphabet->code[i];
        code_s[i] = (std::uint8_t)c;
#pragma unroll
        for (int b = 0; b < bits_; ++b) selectors_s.select[i][b] = ((c >> b) & 1u) ? 0u : 0xFFFFFFFFu;
    }
    __syncthreads();
    int const lane = threadIdx.x & 31;
    std::uint32_t const begin = bins->begin[key_begin];
    std::uint32_t const count = list ? bins->listed[myers_max_words_k + words_]
                                     : bins->begin[key_end - 1] + bins->count[key_end - 1] - begin;
    while (true) {
        std::uint32_t index = 0;
        if (lane == 0) index = atomicAdd(&bins->cursor[key_begin], 1u);
        index = __shfl_sync(0xFFFFFFFFu, index, 0);
        if (index >= count) break;
        pair_task_t const task = tasks[list ? list[begin + index] : begin + index];
        std::uint32_t const distance = myers_warp_distance<words_, bits_>(task, code_s, &selectors_s);
        if (lane == 0) results[task.slot] = distance;
    }
}

/** The same over strings of 16-bit codes (UTF-8 calls over more than 256 code points): 16 planes, no tables. */
template <int words_>
__global__ void __launch_bounds__(256, words_ <= 5 ? 2 : 1) myers_warp_wide_kernel(pair_task_t const *__restrict__ tasks,
                                                              plan_bins_t *__restrict__ bins, int key_begin,
                                                              int key_end, std::int64_t *__restrict__ results,
                                                              std::uint32_t const *__restrict__ list) {
    int const lane = threadIdx.x & 31;
    std::uint32_t const begin = bins->begin[key_begin];
    std::uint32_t const count = list ? bins->listed[myers_max_words_k + words_]
                                     : bins->begin[key_end - 1] + bins->count[key_end - 1] - begin;
    while (true) {
        std::uint32_t index = 0;
        if (lane == 0) index = atomicAdd(&bins->cursor[key_begin], 1u);
        index = __shfl_sync(0xFFFFFFFFu, index, 0);
        if (index >= count) break;
        pair_task_t const task = tasks[list ? list[begin + index] : begin + index];
        std::uint32_t const distance = myers_warp_distance<words_, myers_wide_planes_k, true>(
            task, nullptr, static_cast<plane_selectors_t<myers_wide_planes_k> const *>(nullptr));
        if (lane == 0) results[task.slot] = distance;
    }
}

} // namespace szs_gb300