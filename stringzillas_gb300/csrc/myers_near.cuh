/**
 *  @file myers_near.cuh
 *  @brief Unit-cost Levenshtein distance of similar strings by the bit-parallel method on the blocks around the main
 *         diagonal only, one thread per pair.
 *
 *  A path of cost d from (0, 0) to (n, m), m >= n, never leaves the diagonals from -(d - (m - n)) / 2 to
 *  (d + (m - n)) / 2 (E. Ukkonen, Information and Control 1985), so a distance of at most 64 h - (m - n) is found by
 *  scoring the rows within 32 h of the diagonal. The pattern's 32-row blocks are kept in a window of 2 h + 1 words that
 *  moves down one block every 32 columns (the block form of Myers' algorithm, as in M. Sosic and M. Sikic,
 *  Bioinformatics 2017): at columns 32 c .. 32 c + 31 the window holds blocks c - h .. c + h. Cells outside are replaced
 *  by upper bounds: the row above the window grows by one per column, and a block entering at the bottom starts one
 *  above its upper neighbour in every row. Every value is then the cost of some path, and exact wherever an optimal path
 *  stays inside, so a result of at most 64 h - (m - n) is the distance; any other pair is listed for the full kernel of
 *  its bin (myers_table.cuh, myers.cuh, myers_warp.cuh), which scores it from the start. Pairs far apart give up early:
 *  values on the final diagonal never decrease, so they stop when it passes the limit, or when its growth so far
 *  predicts that it will. Which calls are tried at all is `near_pays`' choice, by the ends of sampled pairs; should nearly
 *  all pairs tried fail for all that (alike at their ends only), the CTAs still to come list theirs untried.
 *
 *  Measured: 1,048,576 DNA pairs of U[100, 300], 4 % apart, 1.22 -> 0.63 ms per call (895,168 of them here in 0.50 ms,
 *  bound by the integer pipe: 34 operations a column for three words); 4,096 reads of 1,000-4,000 2.03 -> 0.78 ms (nine
 *  words, bound by each thread's own chain: one warp per scheduler); 65,536 CJK pairs of 100-300 code points 1.07 ->
 *  0.22 ms of scoring. Unrelated batches are not tried (the planner's sample), at the same time as before.
 *
 *  Work per column: 2 h + 1 words instead of n / 32. Match masks: DNA-like batches (at most four codes) keep the
 *  window's masks of each code in shared memory, 16 bytes per thread, code and four words, moved by one word per block;
 *  other byte strings keep 8 bit planes of the window's bytes in registers, 16-bit codes 16 planes.
 */
#pragma once
#include "myers.cuh"
#include "myers_table.cuh"

namespace szs_gb300 {

enum near_mode_t : int {
    near_dna_k = 0,   // at most four codes: masks in shared memory
    near_bytes_k = 1, // any bytes: 8 planes
    near_wide_k = 2,  // 16-bit codes: 16 planes
};

constexpr int near_threads_k = 128;

/** Dynamic shared memory of one CTA: the DNA form's masks. */
__host__ __device__ constexpr int near_shared_bytes(int half, int mode) {
    return mode == near_dna_k ? myers_table_shared_bytes(2 * half + 1) : 0;
}

/** Transposes the bit matrices of side `side_` in the lanes of `side_` bits of words x[0 .. side_): afterwards bit i of
 *  a lane of x[b] is what bit b of that lane of x[i] was. */
template <int side_, int s_ = side_ / 2>
__device__ __forceinline__ void transpose_bits(std::uint32_t (&x)[side_]) {
    // The low s_ bits of every group of 2 s_.
    constexpr std::uint32_t mask = s_ == 8 ? 0x00FF00FFu : s_ == 4 ? 0x0F0F0F0Fu : s_ == 2 ? 0x33333333u : 0x55555555u;
#pragma unroll
    for (int i = 0; i < side_; ++i) {
        if (i & s_) continue;
        std::uint32_t const t = ((x[i] >> s_) ^ x[i + s_]) & mask;
        x[i + s_] ^= t;
        x[i] ^= t << s_;
    }
    if constexpr (s_ > 1) transpose_bits<side_, s_ / 2>(x);
}

/** The window of blocks of one pair and its step over one text symbol. */
template <int half_>
struct near_window_t {
    static constexpr int B = 2 * half_ + 1;
    std::uint32_t pv[B], mv[B];

    __device__ __forceinline__ void step(std::uint32_t const *eq) {
        std::uint32_t xv[B], sum[B];
#pragma unroll
        for (int w = 0; w < B; ++w) {
            xv[w] = eq[w] | mv[w];
            sum[w] = eq[w] & pv[w];
        }
        asm volatile("add.cc.u32 %0, %0, %1;" : "+r"(sum[0]) : "r"(pv[0]));
#pragma unroll
        for (int w = 1; w < B; ++w) asm volatile("addc.cc.u32 %0, %0, %1;" : "+r"(sum[w]) : "r"(pv[w]));
        std::uint32_t ph_prev = 1u << 31, mh_prev = 0u; // +1 into the row above the window
#pragma unroll
        for (int w = 0; w < B; ++w) {
            std::uint32_t const xh = (sum[w] ^ pv[w]) | eq[w];
            std::uint32_t const ph = mv[w] | ~(xh | pv[w]);
            std::uint32_t const mh = pv[w] & xh;
            std::uint32_t const ph_shifted = __funnelshift_l(ph_prev, ph, 1);
            std::uint32_t const mh_shifted = __funnelshift_l(mh_prev, mh, 1);
            pv[w] = mh_shifted | ~(xv[w] | ph_shifted);
            mv[w] = ph_shifted & xv[w];
            ph_prev = ph, mh_prev = mh;
        }
    }
    /** Moves the window down one block; returns what the value above it grows by. */
    __device__ __forceinline__ std::int32_t advance() {
        std::int32_t const grown = __popc(pv[0]) - __popc(mv[0]);
#pragma unroll
        for (int w = 0; w + 1 < B; ++w) pv[w] = pv[w + 1], mv[w] = mv[w + 1];
        pv[B - 1] = 0xFFFFFFFFu, mv[B - 1] = 0u;
        return grown;
    }
    /** Sum of the vertical deltas of the window's first `rows` rows (1 .. 32 B). */
    __device__ __forceinline__ std::int32_t sum_rows(std::uint32_t rows) const {
        std::int32_t total = 0;
#pragma unroll
        for (int w = 0; w < B; ++w) {
            std::uint32_t const base = 32u * w;
            std::uint32_t const mask = rows >= base + 32u ? 0xFFFFFFFFu : (rows > base ? (1u << (rows - base)) - 1u : 0u);
            total += __popc(pv[w] & mask) - __popc(mv[w] & mask);
        }
        return total;
    }
};

/** The class of a pair's full kernel: its words on the thread route, 16 + words per lane on the warp route; and the
 *  first bin key of that class. */
__device__ __forceinline__ int near_class(std::uint32_t n, bool wide, int &first_key) {
    std::uint32_t const thread_words = wide ? (std::uint32_t)myers_wide_max_words_k : (std::uint32_t)myers_max_words_k;
    std::uint32_t const words = (n + 31u) / 32u;
    if (words <= thread_words) {
        first_key = bin_myers_begin_k + (int)words * 16;
        return (int)words;
    }
    int const per_lane = int((n + 1023u) / 1024u);
    first_key = bin_myers_warp_begin_k + (myers_warp_max_words_k - per_lane) * myers_warp_classes_k;
    return myers_max_words_k + per_lane;
}

/** Thread-per-pair kernel over bins [key_begin, key_end), longest patterns first on the thread route's keys. */
template <int half_, int mode_>
__global__ void __launch_bounds__(near_threads_k)
    myers_near_kernel(pair_task_t const *__restrict__ tasks, plan_bins_t *__restrict__ bins, int key_begin, int key_end,
                      batch_alphabet_t const *__restrict__ alphabet, std::int64_t *__restrict__ results,
                      std::uint32_t *__restrict__ list) {
    constexpr int B = 2 * half_ + 1, Q = (B + 3) / 4;
    constexpr bool dna = mode_ == near_dna_k, wide = mode_ == near_wide_k;
    constexpr int P = wide ? 16 : 8;
    constexpr unsigned code_stride = near_threads_k * 16, group_stride = myers_table_symbols_k * near_threads_k * 16;
    extern __shared__ __align__(16) unsigned char near_masks_s[];
    __shared__ std::uint32_t offset_s[dna ? 256 : 1]; // byte -> code * code_stride, as in myers_table.cuh
    __shared__ std::uint8_t code_s[dna ? 256 : 1];
    __shared__ bool give_up_s;
    if constexpr (dna)
        for (int i = threadIdx.x; i < 256; i += blockDim.x) {
            std::uint32_t const c = alphabet->code[i] & (myers_table_symbols_k - 1);
            bool const known = (alphabet->present[i >> 5] >> (i & 31)) & 1u;
            code_s[i] = known ? (std::uint8_t)c : (std::uint8_t)myers_table_unknown_k;
            offset_s[i] = known ? c * code_stride : myers_table_unknown_k;
        }
    unsigned char *const mine = near_masks_s + threadIdx.x * 16u;
    std::uint32_t const begin = bins->begin[key_begin];
    std::uint32_t const count = bins->begin[key_end - 1] + bins->count[key_end - 1] - begin;
    for (std::uint32_t round = blockIdx.x * blockDim.x; round < count; round += gridDim.x * blockDim.x) {
        if (threadIdx.x == 0) {
            std::uint32_t const tried = __ldcg(&bins->near_tried), failed = __ldcg(&bins->near_failed);
            give_up_s = tried >= near_trial_k && failed >= tried / 16u * 15u;
        }
        __syncthreads();
        bool const give_up = give_up_s;
        std::uint32_t const index = round + threadIdx.x;
        bool const live = index < count;
        bool found = false;
        std::uint32_t const at = begin + count - 1u - (live ? index : 0u);
        pair_task_t const task = tasks[at];
        std::uint32_t const n = task.rows_length, m = task.cols_length, delta = m - n;
        std::int32_t const limit = 64 * half_ - (std::int32_t)delta;
        if (live && !give_up && delta <= 32u * half_) {
            // The text, four symbols' worth of bytes at a time from aligned words (never past the one holding its last
            // byte), shifted to its own alignment.
            std::uint32_t const text_bytes = wide ? 2u * m : m;
            std::uintptr_t const text_address = reinterpret_cast<std::uintptr_t>(task.cols);
            std::uint32_t const *text = reinterpret_cast<std::uint32_t const *>(text_address & ~std::uintptr_t(3));
            std::uint32_t const text_skew = (std::uint32_t)(text_address & 3);
            std::uint32_t const text_last = (text_skew + text_bytes - 1) >> 2;
            std::uint32_t low = __ldg(text), high = text_last >= 1 ? __ldg(text + 1) : 0u;
            std::uint32_t word = 0; // words of the text consumed
            auto next_text = [&]() -> std::uint32_t {
                std::uint32_t const four = __funnelshift_r(low, high, 8 * text_skew);
                low = high;
                if (word + 2 <= text_last) high = __ldg(text + word + 2);
                ++word;
                return four;
            };
            // 32 rows of the pattern as words of bytes, realigned; rows past its end read its first symbol.
            std::uint32_t const pattern_bytes = wide ? 2u * n : n;
            std::uintptr_t const pattern_address = reinterpret_cast<std::uintptr_t>(task.rows);
            std::uint32_t const *pattern = reinterpret_cast<std::uint32_t const *>(pattern_address & ~std::uintptr_t(3));
            std::uint32_t const skew = (std::uint32_t)(pattern_address & 3);
            std::uint32_t const last = (skew + pattern_bytes - 1) >> 2;
            constexpr int words = wide ? 16 : 8; // per block
            std::uint32_t seen = 0; // the marker bit of bytes outside a guessed alphabet
            std::uint32_t filler = wide ? (std::uint32_t)*reinterpret_cast<std::uint16_t const *>(task.rows) * 0x00010001u
                                        : (std::uint32_t)*task.rows * 0x01010101u;
            auto block_words = [&](std::uint32_t block, std::uint32_t (&r)[words]) {
                std::uint32_t v[words + 1];
                std::uint32_t const first = block * words;
#pragma unroll
                for (int i = 0; i <= words; ++i) v[i] = __ldg(pattern + min(first + i, last));
#pragma unroll
                for (int i = 0; i < words; ++i) {
                    r[i] = __funnelshift_r(v[i], v[i + 1], 8 * skew);
                    int const keep = (int)pattern_bytes - 4 * (int)(first + i); // bytes of r[i] inside the pattern
                    std::uint32_t const mask = keep >= 4 ? 0xFFFFFFFFu : (keep <= 0 ? 0u : 0xFFFFFFFFu >> (32 - 8 * keep));
                    r[i] = (r[i] & mask) | (filler & ~mask);
                }
            };

            near_window_t<half_> window;
            [[maybe_unused]] std::uint32_t planes[dna ? 1 : P][dna ? 1 : B];
#pragma unroll
            for (int w = 0; w < B; ++w) window.pv[w] = w < half_ ? 0u : 0xFFFFFFFFu, window.mv[w] = 0u;
            if constexpr (dna) {
#pragma unroll
                for (int q = 0; q < Q; ++q)
#pragma unroll
                    for (int c = 0; c < myers_table_symbols_k; ++c)
                        *reinterpret_cast<uint4 *>(mine + c * code_stride + q * group_stride) = make_uint4(0, 0, 0, 0);
            }
            else {
#pragma unroll
                for (int b = 0; b < P; ++b)
#pragma unroll
                    for (int w = 0; w < B; ++w) planes[b][w] = 0u;
            }
            // Words above the pattern's first row match nothing (planes of zeros would match the symbol 0).
            [[maybe_unused]] std::uint32_t gate[half_];
#pragma unroll
            for (int w = 0; w < half_; ++w) gate[w] = 0u;
            // Takes a block of the pattern in as the window's last word, the others moving up one. Blocks above the
            // pattern (before the first) hold no deltas and no matches, so they pass +1 through.
            auto take_block = [&](std::uint32_t block) {
                std::uint32_t r[words];
                block_words(block, r);
                if constexpr (dna) {
                    std::uint32_t halves[2];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        std::uint32_t x = 0; // row 16 h + k's code at bits 2k (plane 0) and 2k + 1 (plane 1)
#pragma unroll
                        for (int k = 15; k >= 0; --k) {
                            std::uint32_t const code = code_s[__byte_perm(r[4 * h + k / 4], 0u, 0x4440u + (k & 3))];
                            x = x * 4u + code;
                            seen |= code;
                        }
                        // Unshuffle: even bits to the low half, odd bits to the high half.
                        std::uint32_t t;
                        t = (x ^ (x >> 1)) & 0x22222222u, x ^= t ^ (t << 1);
                        t = (x ^ (x >> 2)) & 0x0C0C0C0Cu, x ^= t ^ (t << 2);
                        t = (x ^ (x >> 4)) & 0x00F000F0u, x ^= t ^ (t << 4);
                        t = (x ^ (x >> 8)) & 0x0000FF00u, x ^= t ^ (t << 8);
                        halves[h] = x;
                    }
                    std::uint32_t const a0 = __byte_perm(halves[0], halves[1], 0x5410u);
                    std::uint32_t const a1 = __byte_perm(halves[0], halves[1], 0x7632u);
#pragma unroll
                    for (int c = 0; c < myers_table_symbols_k; ++c) {
                        std::uint32_t const mask = (a0 ^ ((c & 1) ? 0u : ~0u)) & (a1 ^ ((c & 2) ? 0u : ~0u));
                        std::uint32_t words4[4 * Q + 1];
#pragma unroll
                        for (int q = 0; q < Q; ++q) {
                            uint4 const v = *reinterpret_cast<uint4 const *>(mine + c * code_stride + q * group_stride);
                            words4[4 * q] = v.x, words4[4 * q + 1] = v.y, words4[4 * q + 2] = v.z, words4[4 * q + 3] = v.w;
                        }
                        words4[B] = mask;
#pragma unroll
                        for (int q = 0; q < Q; ++q)
                            *reinterpret_cast<uint4 *>(mine + c * code_stride + q * group_stride) =
                                make_uint4(words4[4 * q + 1], 4 * q + 2 <= B ? words4[4 * q + 2] : 0u,
                                           4 * q + 3 <= B ? words4[4 * q + 3] : 0u,
                                           4 * q + 4 <= B ? words4[4 * q + 4] : 0u);
                    }
                }
                else {
                    // The block's bit planes: words ordered so that transposing the small matrices in their lanes leaves
                    // row k at bit k of every plane.
                    std::uint32_t x[P];
                    if constexpr (wide) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) // rows i and i + 16
                            x[i] = __byte_perm(r[i / 2], r[i / 2 + 8], (i & 1) ? 0x7632u : 0x5410u);
                    }
                    else {
#pragma unroll
                        for (int i = 0; i < 8; ++i) { // rows i, i + 8, i + 16 and i + 24
                            std::uint32_t const pick = 0x0040u + 0x0011u * (i & 3);
                            x[i] = __byte_perm(__byte_perm(r[i / 4], r[i / 4 + 2], pick),
                                               __byte_perm(r[i / 4 + 4], r[i / 4 + 6], pick), 0x5410u);
                        }
                    }
                    transpose_bits(x);
#pragma unroll
                    for (int b = 0; b < P; ++b) {
#pragma unroll
                        for (int w = 0; w + 1 < B; ++w) planes[b][w] = planes[b][w + 1];
                        planes[b][B - 1] = x[b];
                    }
                }
            };
            auto column = [&](std::uint32_t symbol) {
                std::uint32_t eq[dna ? 4 * Q : B];
                if constexpr (dna) {
                    std::uint32_t const offset = offset_s[symbol];
                    seen |= offset;
#pragma unroll
                    for (int q = 0; q < Q; ++q) {
                        uint4 const v = *reinterpret_cast<uint4 const *>(mine + offset + q * group_stride);
                        eq[4 * q] = v.x, eq[4 * q + 1] = v.y, eq[4 * q + 2] = v.z, eq[4 * q + 3] = v.w;
                    }
                }
                else {
#pragma unroll
                    for (int w = 0; w < B; ++w) eq[w] = w < half_ ? gate[w] : 0xFFFFFFFFu;
#pragma unroll
                    for (int b = 0; b < P; ++b) {
                        std::uint32_t const select = ((symbol >> b) & 1u) - 1u; // all ones where the bit is 0
#pragma unroll
                        for (int w = 0; w < B; ++w) eq[w] &= planes[b][w] ^ select;
                    }
                }
                window.step(eq);
            };

            for (int block = 0; block < half_; ++block) take_block(block);
            std::int32_t above = 0; // the value of the row above the window
            std::uint32_t done = 0; // columns scored
            bool alive = true;
            while (true) {
                take_block((done >> 5) + half_);
                if (done + 32u > m) break;
                constexpr int per_word = wide ? 2 : 4;
#pragma unroll 1
                for (int four = 0; four < 32 / per_word; ++four) {
                    std::uint32_t const symbols = next_text();
#pragma unroll
                    for (int k = 0; k < per_word; ++k)
                        column(wide ? (k ? symbols >> 16 : symbols & 0xFFFFu) : __byte_perm(symbols, 0u, 0x4440u + k));
                }
                done += 32u, above += 32;
                if (done == m) break;
                // The final diagonal's value here: it can only grow from now on, and strings that differ in more than a
                // third of their symbols so far, or more often than the limit allows (with some room for chance), are
                // given up. Unrelated DNA differs in about 17 of the first 32, a fifth of substitutions in 6 or 7.
                std::int32_t const value = above + window.sum_rows(32u * (half_ + 1) - delta);
                std::int32_t const edits = max(value - (std::int32_t)delta, 0); // beyond those of the unequal lengths
                float const grown = (float)edits - 3.0f - 1.5f * sqrtf((float)edits);
                alive = value <= limit && 3 * edits <= (std::int32_t)done + 8 &&
                        grown * (float)m <= (float)limit * (float)done;
                if (!alive) break;
                above += window.advance();
#pragma unroll
                for (int w = 0; w < half_; ++w) gate[w] = w + 1 < half_ ? gate[w + 1] : 0xFFFFFFFFu;
            }
            if (alive) {
                constexpr int per_word = wide ? 2 : 4;
                std::uint32_t const before = done; // columns of whole blocks
                while (done < m) {
                    std::uint32_t symbols = next_text();
                    std::uint32_t const here = min((std::uint32_t)per_word, m - done);
                    for (std::uint32_t k = 0; k < here; ++k) {
                        column(symbols & (wide ? 0xFFFFu : 0xFFu));
                        symbols >>= wide ? 16 : 8;
                    }
                    done += here;
                }
                above += (std::int32_t)(m - before);
                std::uint32_t const top = (m - 1u) >> 5; // the last column's block; the window starts half_ blocks higher
                std::int32_t const score = above + window.sum_rows(n + 32u * half_ - 32u * top);
                found = score <= limit;
                if (found) {
                    results[task.slot] = score;
                    if (seen & myers_table_unknown_k) atomicOr(&bins->error_flags, 2u);
                }
            }
        }
        // The lanes of a warp with pairs of one class to list take their places with one atomic.
        int first_key = 0;
        int const which = live && !found ? near_class(n, wide, first_key) : -1;
        unsigned const peers = __match_any_sync(0xFFFFFFFFu, which);
        if (which >= 0) {
            int const lane = threadIdx.x & 31, leader = __ffs(peers) - 1;
            std::uint32_t place = 0;
            if (lane == leader) place = atomicAdd(&bins->listed[which], (std::uint32_t)__popc(peers));
            place = __shfl_sync(peers, place, leader);
            list[bins->begin[first_key] + place + __popc(peers & ((1u << lane) - 1u))] = at;
        }
        int const failed = __syncthreads_count(live && !found && !give_up);
        if (threadIdx.x == 0 && !give_up) {
            atomicAdd(&bins->near_tried, min(count - round, (std::uint32_t)blockDim.x));
            if (failed) atomicAdd(&bins->near_failed, (std::uint32_t)failed);
        }
    }
}

} // namespace szs_gb300
