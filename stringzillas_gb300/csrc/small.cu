/**
 *  @file small.cu
 *  @brief Small pairwise calls of unit-cost Levenshtein from host memory: one copy, one kernel, results written to host
 *         memory.
 *
 *  A call of a few hundred short pairs spends its time around the scoring: four copies of tapes and offsets, the alphabet
 *  and planning kernels, a round trip for the plan, a launch per word count on forked streams, a result copy. When the
 *  offsets are in host memory the host knows every length, so it packs the strings and one 16-byte record per pair into
 *  one page-locked buffer, and a single kernel scores the pairs, one warp each.
 *
 *  The warp kernel is the one of myers_warp.cuh at one word per lane (patterns of up to 1,024 bytes). A step's time is its
 *  instruction count times the latency of one warp, so what does not depend on the step before is taken off it: each lane
 *  loads its own text byte two steps ahead, and the match mask a step ahead: patterns of up to 256 bytes keep their masks
 *  in shared memory by byte (a warp's match-any over 32 rows gives each distinct byte's mask at once), longer ones form
 *  them from 8 bit planes taken by ballots. No alphabet is needed. The distance comes from the vertical deltas of the
 *  last column. 64 pairs of 64-256 bytes: 33 us with planes and bytes passed from lane to lane, 28 us now.
 */
#include "launchers.h"

#include <algorithm>

namespace szs_gb300 {

namespace {

constexpr int small_warps_k = 4;                  // pairs per CTA
constexpr std::uint32_t small_table_words_k = 8;  // patterns of up to 256 bytes

__global__ void __launch_bounds__(32 * small_warps_k)
    myers_small_kernel(small_pair_t const *__restrict__ pairs, std::uint32_t const count,
                       std::uint8_t const *__restrict__ bytes, std::int64_t *__restrict__ results) {
    __shared__ __align__(16) std::uint32_t masks_s[small_warps_k][256 * small_table_words_k];
    std::uint32_t const index = blockIdx.x * small_warps_k + threadIdx.x / 32;
    if (index >= count) return;
    int const lane = threadIdx.x & 31;
    small_pair_t const pair = pairs[index];
    std::uint32_t const n = pair.rows_length, m = pair.cols_length;
    std::uint8_t const *rows = bytes + pair.rows, *cols = bytes + pair.cols;
    if (n == 0) {
        if (lane == 0) results[index] = m;
        return;
    }
    std::uint32_t const words = (n + 31u) / 32u;
    std::uint32_t *const masks = masks_s[threadIdx.x / 32];
    bool const tabled = words <= small_table_words_k;
    // The pattern's masks: a table by byte (one word per 32 rows), or lane w's 32 rows as bit planes of their bytes.
    std::uint32_t planes[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (tabled) {
        auto *quads = reinterpret_cast<uint4 *>(masks);
        for (int i = lane; i < 256 * small_table_words_k / 4; i += 32) quads[i] = make_uint4(0, 0, 0, 0);
        __syncwarp();
    }
    for (std::uint32_t w = 0; w < words; ++w) {
        std::uint32_t const row = 32u * w + lane, byte = row < n ? rows[row] : 0u;
        if (tabled) { // rows past the pattern match nothing
            unsigned const same = __match_any_sync(0xFFFFFFFFu, row < n ? byte : 256u);
            if (row < n && lane == __ffs(same) - 1) masks[byte * small_table_words_k + w] = same;
            continue;
        }
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            std::uint32_t const plane = __ballot_sync(0xFFFFFFFFu, (byte >> b) & 1u);
            planes[b] = lane == (int)w ? plane : planes[b];
        }
    }
    __syncwarp();
    std::uint32_t pv = 0xFFFFFFFFu, mv = 0u;
    // At step t lane L scores column t - L.
    std::uint32_t const steps = m + words - 1u;
    auto text = [&](std::uint32_t t) -> std::uint32_t { // lane L's byte of step t (0 outside the text, never scored)
        std::uint32_t const j = t - lane;
        return j < m ? cols[j] : 0u;
    };
    auto sweep = [&](auto &&matches) {
        std::uint32_t eq = matches(text(0)), byte = text(1), out = 0; // out: carry | top Ph bit << 1 | top Mh bit << 2
#pragma unroll 2
        for (std::uint32_t t = 0; t < steps; ++t) {
            std::uint32_t const byte_after = text(t + 2u), eq_next = matches(byte);
            std::uint32_t in = __shfl_up_sync(0xFFFFFFFFu, out, 1);
            if (lane == 0) in = 2u; // no carry into row 0; +1 shifted into its horizontal delta
            if (t - lane < m) {
                std::uint32_t const xv = eq | mv, masked = eq & pv;
                std::uint32_t const partial = masked + pv, sum = partial + (in & 1u);
                std::uint32_t const carry = (partial < masked ? 1u : 0u) | (sum < partial ? 1u : 0u);
                std::uint32_t const xh = (sum ^ pv) | eq, ph = mv | ~(xh | pv), mh = pv & xh;
                std::uint32_t const ph_shifted = ph << 1 | ((in >> 1) & 1u), mh_shifted = mh << 1 | (in >> 2);
                pv = mh_shifted | ~(xv | ph_shifted);
                mv = ph_shifted & xv;
                out = carry | (ph >> 31) << 1 | (mh >> 31) << 2;
            }
            eq = eq_next, byte = byte_after;
        }
    };
    if (tabled) {
        std::uint32_t const *mine = masks + min((std::uint32_t)lane, small_table_words_k - 1u);
        sweep([&](std::uint32_t byte) { return mine[byte * small_table_words_k]; });
    }
    else
        sweep([&](std::uint32_t byte) {
            std::uint32_t eq = 0xFFFFFFFFu;
#pragma unroll
            for (int b = 0; b < 8; ++b) eq &= planes[b] ^ (((byte >> b) & 1u) - 1u);
            return eq;
        });
    // D[n][m] = m + (rows 1..n of the last column's +1 deltas) - (its -1 deltas).
    std::uint32_t const base = 32u * lane;
    std::uint32_t const mask = n >= base + 32u ? 0xFFFFFFFFu : (n > base ? (1u << (n - base)) - 1u : 0u);
    int const total = __reduce_add_sync(0xFFFFFFFFu, __popc(pv & mask) - __popc(mv & mask));
    if (lane == 0) results[index] = (std::int64_t)m + total;
}

} // namespace

cudaError_t launch_myers_small(small_pair_t const *pairs, std::uint32_t count, std::uint8_t const *bytes,
                               std::int64_t *results, cudaStream_t stream) {
    if (!count) return cudaSuccess;
    myers_small_kernel<<<(count + small_warps_k - 1) / small_warps_k, 32 * small_warps_k, 0, stream>>>(pairs, count, bytes,
                                                                                                       results);
    return cudaGetLastError();
}

} // namespace szs_gb300
