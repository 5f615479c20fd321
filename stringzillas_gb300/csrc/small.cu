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
 *  The warp kernel is the one of myers_warp.cuh at one word per lane (patterns of up to 1,024 bytes), but for 8 bit
 *  planes of the bytes themselves, taken by warp ballots, so that no alphabet is needed, and for match masks formed a
 *  step ahead of their use: the text's byte travels from lane to lane one step before the deltas, so only the carried add
 *  and the deltas are on the chain that bounds a step. The distance comes from the vertical deltas of the last column.
 */
#include "launchers.h"

#include <algorithm>

namespace szs_gb300 {

namespace {

constexpr int small_warps_k = 4; // pairs per CTA

__global__ void __launch_bounds__(32 * small_warps_k)
    myers_small_kernel(small_pair_t const *__restrict__ pairs, std::uint32_t const count,
                       std::uint8_t const *__restrict__ bytes, std::int64_t *__restrict__ results) {
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
    // Lane w holds rows 32 w .. 32 w + 31 as bit planes of their bytes.
    std::uint32_t const words = (n + 31u) / 32u;
    std::uint32_t planes[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (std::uint32_t w = 0; w < words; ++w) {
        std::uint32_t const row = 32u * w + lane, byte = row < n ? rows[row] : 0u;
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            std::uint32_t const plane = __ballot_sync(0xFFFFFFFFu, (byte >> b) & 1u);
            planes[b] = lane == (int)w ? plane : planes[b];
        }
    }
    std::uint32_t pv = 0xFFFFFFFFu, mv = 0u;
    auto matches = [&](std::uint32_t byte) {
        std::uint32_t eq = 0xFFFFFFFFu;
#pragma unroll
        for (int b = 0; b < 8; ++b) eq &= planes[b] ^ (((byte >> b) & 1u) - 1u);
        return eq;
    };
    // At step t lane L scores column t - L; its byte came from lane L - 1 a step before, lane 0's from a 32-byte chunk.
    std::uint32_t const steps = m + words - 1u;
    std::uint32_t chunk = (std::uint32_t)lane < m ? cols[lane] : 0u, ahead = 32u + lane < m ? cols[32u + lane] : 0u;
    std::uint32_t byte = __shfl_sync(0xFFFFFFFFu, chunk, 0); // lane 0's first column
    std::uint32_t eq = matches(byte), out = 0;               // out: carry | top Ph bit << 1 | top Mh bit << 2
    for (std::uint32_t t = 0; t < steps; ++t) {
        std::uint32_t const next = t + 1u;
        if ((next & 31u) == 0) chunk = ahead, ahead = next + 32u + lane < m ? cols[next + 32u + lane] : 0u;
        std::uint32_t const staged = __shfl_sync(0xFFFFFFFFu, chunk, int(next & 31u));
        std::uint32_t const passed = __shfl_up_sync(0xFFFFFFFFu, byte, 1);
        std::uint32_t in = __shfl_up_sync(0xFFFFFFFFu, out, 1);
        if (lane == 0) in = 2u; // no carry into row 0; +1 shifted into its horizontal delta
        byte = lane == 0 ? staged : passed;
        std::uint32_t const eq_next = matches(byte);
        int const j = (int)t - lane;
        if (j >= 0 && j < (int)m) {
            std::uint32_t const xv = eq | mv, masked = eq & pv;
            std::uint32_t const partial = masked + pv, sum = partial + (in & 1u);
            std::uint32_t const carry = (partial < masked ? 1u : 0u) | (sum < partial ? 1u : 0u);
            std::uint32_t const xh = (sum ^ pv) | eq, ph = mv | ~(xh | pv), mh = pv & xh;
            std::uint32_t const ph_shifted = ph << 1 | ((in >> 1) & 1u), mh_shifted = mh << 1 | (in >> 2);
            pv = mh_shifted | ~(xv | ph_shifted);
            mv = ph_shifted & xv;
            out = carry | (ph >> 31) << 1 | (mh >> 31) << 2;
        }
        eq = eq_next;
    }
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
