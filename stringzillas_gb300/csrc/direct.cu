/**
 *  @file direct.cu
 *  @brief Cross products under unit-cost Levenshtein: one thread per output cell, a query's match masks shared by the
 *         CTA, no planning.
 *
 *  In a cross product every query meets every candidate, so what the pairwise kernels prepare per pair (code planes or
 *  match masks of the pattern, a task record, a bin) is the same for a whole row of cells. Here a CTA takes one query
 *  as the pattern and a block of candidates: it writes the query's match masks once into a shared table indexed by the
 *  byte itself (no alphabet pass), each thread runs the Myers / Hyyrö step over its candidate with the pattern's deltas
 *  in registers (up to 1,024 rows in 32 words), and writes the distance where it lands in the caller's matrix. A text
 *  column costs one shared load per four words (16-byte loads; rows of the table are an odd number of 16-byte units
 *  apart, so the few letters of a DNA text fall into different banks), and ten integer operations per word, which bound
 *  the kernel: the warp-per-pair kernel spends about 45 on a step of one word per lane.
 *
 *  Measured (device-resident, whole calls): 197 x 198 strings of 1,000 bytes 3.16 ms on the planned warp-per-pair route,
 *  1.01 ms here; 2,048 x 2,048 tokens of 4-16 bytes 0.25 ms with the pattern's bit planes built by every thread, 0.12 ms
 *  here; 197 x 198 of 100 bytes 112 us planned, 52 us here.
 *
 *  Either side may be the pattern, by `direct_choice`, which also leaves calls to the planned routes (direct_rule.h).
 *  Words are chosen per pattern inside a kernel, in steps that fit its class (up to 128, 512 and 1,024 rows), which the
 *  host picks by the longest pattern; classes keep the registers of the long patterns off the short ones.
 *
 *  Counterpart of the reference's single-word direct path for tiny-token cross products
 *  (include/stringzillas/similarities/cuda.cuh:3892-3936); the distances are those of the serial engine
 *  (serial.hpp:1656-1865).
 */
#include "launchers.h"
#include "planner.cuh"

#include <cuda_runtime.h>

#include <algorithm>

namespace szs_gb300 {

namespace {

__device__ __forceinline__ void direct_string(tape_t const &tape, std::uint64_t index, std::uint8_t const *&start,
                                              std::uint64_t &length) {
    std::uint64_t begin, end;
    if (tape.offset_bits == 32) {
        auto const *offsets = static_cast<std::uint32_t const *>(tape.offsets);
        begin = offsets[index], end = offsets[index + 1];
    }
    else {
        auto const *offsets = static_cast<std::uint64_t const *>(tape.offsets);
        begin = offsets[index], end = offsets[index + 1];
    }
    start = tape.base + begin;
    length = tape.lengths ? tape.lengths[index] : end - begin;
}

/** Bytes between two rows of the match-mask table of patterns of `words` words. */
__host__ __device__ constexpr int direct_row_bytes(int words) {
    return words <= 2 ? 4 * words : 16 * (((words + 3) / 4) | 1);
}

/** The unit-cost edit distance of the CTA's pattern (n rows, masks in `table`) and a text of 1 or more bytes. */
template <int words_>
__device__ __forceinline__ std::uint32_t direct_distance(unsigned char const *table, std::uint32_t n,
                                                        std::uint8_t const *text, std::uint32_t m) {
    constexpr int W = words_, Q = (W + 3) / 4;
    std::uint32_t pv[W], mv[W];
#pragma unroll
    for (int w = 0; w < W; ++w) pv[w] = 0xFFFFFFFFu, mv[w] = 0u;
    auto column = [&](std::uint32_t byte) {
        unsigned char const *masks = table + byte * direct_row_bytes(W);
        std::uint32_t eq[4 * Q], xv[W], sum[W];
        if constexpr (W == 1) eq[0] = *reinterpret_cast<std::uint32_t const *>(masks);
        else if constexpr (W == 2) {
            uint2 const v = *reinterpret_cast<uint2 const *>(masks);
            eq[0] = v.x, eq[1] = v.y;
        }
        else {
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                uint4 const v = *reinterpret_cast<uint4 const *>(masks + 16 * q);
                eq[4 * q] = v.x, eq[4 * q + 1] = v.y, eq[4 * q + 2] = v.z, eq[4 * q + 3] = v.w;
            }
        }
#pragma unroll
        for (int w = 0; w < W; ++w) {
            xv[w] = eq[w] | mv[w];
            sum[w] = eq[w] & pv[w];
        }
        // Multi-word (Eq & Pv) + Pv: one add per word, the carry rippling upwards through the carry flag.
        asm volatile("add.cc.u32 %0, %0, %1;" : "+r"(sum[0]) : "r"(pv[0]));
#pragma unroll
        for (int w = 1; w < W; ++w) asm volatile("addc.cc.u32 %0, %0, %1;" : "+r"(sum[w]) : "r"(pv[w]));
        std::uint32_t ph_prev = 1u << 31, mh_prev = 0u; // +1 shifted into row 0
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
    };
    // The text four bytes at a time from aligned words (never past the one holding its last byte), shifted to the
    // text's own alignment so that a warp's lanes step together whatever theirs; the next word is in flight meanwhile.
    std::uintptr_t const address = reinterpret_cast<std::uintptr_t>(text);
    std::uint32_t const *aligned = reinterpret_cast<std::uint32_t const *>(address & ~std::uintptr_t(3));
    std::uint32_t const skew = (std::uint32_t)(address & 3), last = (skew + m - 1) >> 2;
    std::uint32_t low = __ldg(aligned), high = last >= 1 ? __ldg(aligned + 1) : 0u;
    for (std::uint32_t c = 0; c < m / 4; ++c) {
        std::uint32_t const four = __funnelshift_r(low, high, 8 * skew);
        low = high;
        if (c + 2 <= last) high = __ldg(aligned + c + 2);
#pragma unroll
        for (int k = 0; k < 4; ++k) column(__byte_perm(four, 0u, 0x4440u + k));
    }
    std::uint32_t rest = __funnelshift_r(low, high, 8 * skew);
    for (std::uint32_t j = 0; j < (m & 3u); ++j, rest >>= 8) column(rest & 0xFFu);
    // D[n][m] = m + (rows 1..n of the last column's +1 deltas) - (its -1 deltas).
    std::uint32_t distance = m;
#pragma unroll
    for (int w = 0; w < W; ++w) {
        std::uint32_t const base = 32u * w;
        std::uint32_t const mask = n >= base + 32u ? 0xFFFFFFFFu : (n > base ? (1u << (n - base)) - 1u : 0u);
        distance += __popc(pv[w] & mask) - __popc(mv[w] & mask);
    }
    return distance;
}

/** A pattern's row of cells with the fewest words of the class that hold it (`words_`, or steps above). */
template <int words_, int step_, int most_, typename visit_>
__device__ __forceinline__ void direct_with_words(std::uint32_t words, visit_ &&visit) {
    if constexpr (words_ + step_ <= most_)
        if (words > words_) return direct_with_words<words_ + step_, step_, most_>(words, visit);
    visit(std::integral_constant<int, words_> {});
}

/**
 *  One pattern per CTA and round, one cell per thread and round: patterns along the grid's y dimension, texts along x.
 *  `swapped`: the patterns are the candidates.
 */
template <int first_, int step_, int most_>
__global__ void __launch_bounds__(256, most_ <= 4 ? 5 : (most_ <= 16 ? 3 : 2))
    myers_direct_kernel(tape_t const patterns, tape_t const texts, int const swapped, std::int64_t *__restrict__ out,
                        std::uint64_t const stride) {
    extern __shared__ __align__(16) unsigned char masks_s[];
    for (std::uint64_t p = blockIdx.y; p < patterns.count; p += gridDim.y) {
        std::uint8_t const *pattern;
        std::uint64_t n;
        direct_string(patterns, p, pattern, n);
        direct_with_words<first_, step_, most_>((std::uint32_t)((n + 31) / 32), [&](auto words) {
            constexpr int W = decltype(words)::value;
            constexpr int row_words = direct_row_bytes(W) / 4;
            auto *table = reinterpret_cast<std::uint32_t *>(masks_s);
            __syncthreads(); // the previous pattern's readers are done
            for (std::uint32_t i = threadIdx.x; i < 256u * row_words; i += blockDim.x) table[i] = 0u;
            __syncthreads();
            for (std::uint32_t i = threadIdx.x; i < n; i += blockDim.x)
                atomicOr(&table[(std::uint32_t)pattern[i] * row_words + (i >> 5)], 1u << (i & 31u));
            __syncthreads();
            for (std::uint64_t t = (std::uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < texts.count;
                 t += (std::uint64_t)gridDim.x * blockDim.x) {
                std::uint8_t const *text;
                std::uint64_t m;
                direct_string(texts, t, text, m);
                std::uint32_t const distance =
                    n && m ? direct_distance<W>(masks_s, (std::uint32_t)n, text, (std::uint32_t)m)
                           : (std::uint32_t)(n + m);
                out[swapped ? t * stride + p : p * stride + t] = distance;
            }
        });
    }
}

/** One part of a tape per CTA (queries for blockIdx.y 0, candidates for 1), straight into page-locked host memory. The
 *  call waits for it, so its reductions are few: what a group of 32 strings shares is the same in all lanes as it is, and
 *  the sums of words, which only choose a route, have 32 bits per warp (2,048 x 2,048 tokens: 120 us a call with seven sums
 *  in 64 bits and atomics, 117 this way). */
__global__ void __launch_bounds__(1024) direct_extents_kernel(tape_t const queries, tape_t const candidates,
                                                              int const query_parts, int const candidate_parts,
                                                              direct_extents_t *__restrict__ extents) {
    int const parts = blockIdx.y ? candidate_parts : query_parts;
    if ((int)blockIdx.x >= parts) return;
    constexpr int fields = sizeof(direct_extents_t) / 8;
    __shared__ unsigned long long warps_s[fields][32];
    int const lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    tape_t const &tape = blockIdx.y ? candidates : queries;
    unsigned long long symbols = 0, padded = 0;
    std::uint32_t longest = 0, words = 0, to_two = 0, to_four = 0, long_words = 0;
    // A warp takes 32 strings at a time, the group that a warp of the direct kernels would.
    std::uint64_t const threads = (std::uint64_t)parts * blockDim.x;
    std::uint64_t const rounded = (tape.count + 31) / 32 * 32;
#pragma unroll 8
    for (std::uint64_t i = (std::uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < rounded; i += threads) {
        std::uint8_t const *start;
        std::uint64_t length = 0;
        if (i < tape.count) direct_string(tape, i, start, length);
        std::uint32_t const most = __reduce_max_sync(0xFFFFFFFFu, (std::uint32_t)min(length, (std::uint64_t)0xFFFFFFFFu));
        std::uint32_t const here = (std::uint32_t)((length + 31) / 32);
        longest = max(longest, most);
        symbols += length, padded += 32ull * most;
        words += here, to_two += here & 1u, to_four += (0u - here) & 3u;
        long_words += length > 512 ? here : 0u;
    }
    unsigned long long const low = __reduce_add_sync(0xFFFFFFFFu, (std::uint32_t)symbols & 0xFFFFu);
    unsigned long long const high = __reduce_add_sync(0xFFFFFFFFu, (std::uint32_t)(symbols >> 16));
    words = __reduce_add_sync(0xFFFFFFFFu, words), to_two = __reduce_add_sync(0xFFFFFFFFu, to_two);
    to_four = __reduce_add_sync(0xFFFFFFFFu, to_four), long_words = __reduce_add_sync(0xFFFFFFFFu, long_words);
    if (lane == 0) {
        warps_s[0][warp] = longest, warps_s[1][warp] = (high << 16) + low, warps_s[2][warp] = padded;
        warps_s[3][warp] = words, warps_s[4][warp] = (unsigned long long)words + to_two;
        warps_s[5][warp] = (unsigned long long)words + to_four, warps_s[6][warp] = long_words;
    }
    __syncthreads();
    if (warp >= fields) return;
    unsigned long long value = warps_s[warp][lane];
#pragma unroll
    for (int distance = 16; distance; distance >>= 1) {
        unsigned long long const other = __shfl_xor_sync(0xFFFFFFFFu, value, distance);
        value = warp == 0 ? max(value, other) : value + other;
    }
    if (lane == 0)
        reinterpret_cast<unsigned long long *>(extents + (blockIdx.y ? query_parts : 0) + blockIdx.x)[warp] = value;
}

} // namespace

cudaError_t launch_direct_extents(tape_t const &queries, tape_t const &candidates, direct_extents_t *extents,
                                  cudaStream_t stream) {
    int const query_parts = direct_extents_parts(queries.count), candidate_parts = direct_extents_parts(candidates.count);
    dim3 const grid(std::max(query_parts, candidate_parts), 2);
    direct_extents_kernel<<<grid, 1024, 0, stream>>>(queries, candidates, query_parts, candidate_parts, extents);
    return cudaGetLastError();
}

cudaError_t launch_myers_direct(tape_t const &queries, tape_t const &candidates, bool swapped, std::uint64_t longest_rows,
                                std::int64_t *out, std::uint64_t stride, int sm_count, cudaStream_t stream) {
    tape_t const &patterns = swapped ? candidates : queries, &texts = swapped ? queries : candidates;
    // Small CTAs while there are few cells for the SMs, so that the last round is even; larger ones share a pattern's
    // table among more threads.
    unsigned threads = 256;
    while (threads > 64 && (threads / 2 >= texts.count ||
                            patterns.count * ((texts.count + threads - 1) / threads) < (std::uint64_t)sm_count * 8))
        threads /= 2;
    // A CTA's table serves several rounds of texts when the patterns alone make enough CTAs (about four waves of five per
    // SM): 2,048 x 2,048 tokens take 123 us with a table per 256 cells, 116 us with one per 1,024.
    std::uint64_t const columns = (texts.count + threads - 1) / threads;
    std::uint64_t const across = ((std::uint64_t)sm_count * 20 + patterns.count - 1) / patterns.count;
    unsigned const grid_x = (unsigned)std::min<std::uint64_t>(columns, across);
    std::uint64_t const wanted = ((std::uint64_t)sm_count * 32 + grid_x - 1) / grid_x;
    unsigned const grid_y = (unsigned)std::min<std::uint64_t>({patterns.count, wanted, 65535});
    dim3 const grid(grid_x, grid_y);
    int const set = swapped ? 1 : 0;
    if (longest_rows <= 128)
        myers_direct_kernel<1, 1, 4><<<grid, threads, 256 * direct_row_bytes(4), stream>>>(patterns, texts, set, out,
                                                                                          stride);
    else if (longest_rows <= 512)
        myers_direct_kernel<2, 2, 16><<<grid, threads, 256 * direct_row_bytes(16), stream>>>(patterns, texts, set, out,
                                                                                            stride);
    else
        myers_direct_kernel<4, 4, 32><<<grid, threads, 256 * direct_row_bytes(32), stream>>>(patterns, texts, set, out,
                                                                                            stride);
    return cudaGetLastError();
}

} // namespace szs_gb300
