/**
 *  @file planner.cuh
 *  @brief Device-side planning of one batch: enumerate the pairs of a call, answer the trivial ones, choose a
 *         route and a length bin for the rest, and counting-sort them into bins.
 *
 *  The reference does this with a materialisation kernel, a min/max probe, a histogram, a scan and a scatter,
 *  syncing the host between stages (include/stringzillas/similarities/cuda.cuh:1583-1747, :1859-1914). Here the
 *  whole plan stays on the device: three kernels, no host round trip until the launch list is read back, and
 *  bins are ordered so persistent kernels meet the longest pairs first (longest-processing-time order).
 *
 *  Bin keys:
 *    [0, 272)    Myers: key = words * 16 + text-length class (words 1..16)
 *    [272, 304)  32-bit wavefront DP: key = 272 + (31 - size class), size class ~ log2(n * m)
 *    [304, 336)  64-bit wavefront DP: same layout
 *    [336, 1360) 16x2 packed wavefront DP: key = 336 + 256 * rows-per-lane index + 8 * (31 - n class)
 *                + (7 - ratio class), n class = 4 log2(n) - 12 (quarter octaves of the shorter side), ratio class
 *                = 2 log2(m / n); rows per lane R in {4, 8, 12, 16}, chosen per pair. A warp scores two consecutive
 *                pairs of a bin at once and pays for the larger of each dimension, so bins are narrow in both.
 *    [1360, 1392) band (one CTA per pair, 32-bit cells): key = 1360 + (31 - size class), size class ~ log2(n * m)
 *    [1392, 1424) 16-bit band (one CTA per pair, 16x2 cells): same layout from 1392
 *    [1424, 1488) warp-per-pair Myers (unit Levenshtein, shorter side 513..8,192): key = 1424 + 8 * (8 - W)
 *                 + (7 - text class), W = words per lane = ceil(n / 1024), text class ~ log2(m) - 9
 *    [1488, 2028) short pairs on 16x2 cells (shorter side <= 448): key = 1488 + 27 * shape + (26 - m class), shape 0 for
 *                 n <= 16, then four per octave (`short_segment_rows`), m class = excess / 16 below 320, then
 *                 20 + log2(excess) - 8, excess = m - rows of the next smaller shape
 *    2028         unit-cost Levenshtein beyond the warp kernel (shorter side 8,193 .. 2^20): a chain of warps per pair
 */
#pragma once
#include "engine_types.cuh"

namespace szs_gb300 {

constexpr int bin_keys_k = 2048;
constexpr int bin_myers_begin_k = 0;
constexpr int bin_dp32_begin_k = 272;
constexpr int bin_dp64_begin_k = 304;
constexpr int bin_dp16_begin_k = 336;
constexpr int bin_dp_classes_k = 32;
constexpr int bin_dp16_classes_k = 1024;
constexpr int dp16_row_choices_k = 4;       // rows per lane 4, 8, 12, 16
constexpr int dp16_classes_per_rows_k = 256; // shape classes within one rows-per-lane choice (32 n x 8 ratio)
constexpr int bin_band_begin_k = bin_dp16_begin_k + bin_dp16_classes_k; // 1360
constexpr int bin_band16_begin_k = bin_band_begin_k + bin_dp_classes_k;  // 1392
static_assert(bin_band16_begin_k + bin_dp_classes_k <= bin_keys_k, "bin layout exceeds the key space");
static_assert(bin_keys_k % 2 == 0 && bin_keys_k / 2 <= 1024, "the scan kernel uses one CTA of bin_keys_k / 2 threads");
constexpr int band_min_rows_k = 1024;        // default: 32-bit pairs whose shorter side exceeds this take a whole CTA
/** Built-in relative costs of one lane step of the 16x2 route with 4, 8, 12, 16 rows per lane, measured on GB300
 *  (affine protein alignment, shorter sides 128-1,023). */
constexpr int packed_step_cost_k[4] = {100, 165, 245, 330};
constexpr int band_min_rows_packed_k = 2048; // default for pairs that fit 16-bit cells (the 16-bit band above it)
constexpr int band_min_rows_few_k = 1024;    // default for calls with fewer pairs than one 16x2 wave (32 per SM)
constexpr int band_min_rows_compare_k = 2048; // default for compare-mode Levenshtein pairs on 16-bit cells
constexpr int myers_max_words_k = 16;
constexpr int myers_wide_max_words_k = 8; // 16-bit codes take 16 code planes: the thread route stops at 8 words
// Words per lane of the warp kernel: patterns up to 32 * 32 * 8 = 8,192 rows. Longer ones take the bands: a pair of
// 8-16k characters keeps one warp busy for milliseconds, and a call rarely has enough of them to fill the GPU.
constexpr int myers_warp_max_words_k = 8;
constexpr int myers_warp_classes_k = 8;    // text-length classes per words count (longest first)
constexpr int bin_myers_warp_begin_k = bin_band16_begin_k + bin_dp_classes_k; // 1424
static_assert(bin_myers_warp_begin_k + myers_warp_max_words_k * myers_warp_classes_k <= bin_keys_k,
              "bin layout exceeds the key space");
constexpr int bin_short_begin_k = bin_myers_warp_begin_k + myers_warp_max_words_k * myers_warp_classes_k; // 1488
constexpr int short_shapes_k = 20;     // segments holding 16 rows, then four shapes per octave up to 448
constexpr int short_m_classes_k = 27;  // text-length classes per shape
constexpr int short_max_rows_k = 448;  // default: shorter sides up to this take the short route (large batches)
constexpr int short_few_rows_k = 128;  // the same for smaller batches and the plain form
constexpr int short_profile_rows_k = 192; // the same for large batches whose profile has many classes
constexpr int short_row_maxima_k = 3;  // beside the compare modes: local scores with positive gap costs (dp_short.cuh)
constexpr std::uint64_t short_row_maxima_pairs_k = 12288; // pairs from which those take the short route
constexpr int short_few_classes_k = 8; // profiles over at most this many classes fit segments of 16-28 rows per lane
/** Pairs, and cells by the mean sides of 32 of them, from which a call cuts its short pairs' rows in quarter octaves
 *  instead of halves and takes longer ones: 655e6 cells of text pairs of 100-300 took 334 us either way (340 here), 800e6 384 -> 370
 *  and 1.3e9 573 -> 515; 340e6 cells of DNA pairs of 16-128 226 -> 263. */
constexpr std::uint64_t short_fine_pairs_k = 1 << 14;
constexpr float short_fine_cells_k = 800e6f;
/** Rows of all pairs together that such a call needs besides, by the means of the shorter and the longer sides: a warp
 *  holds some 1,500 rows in quarter octaves, half as many in halves, and a call of few warps, spread over many shapes, takes
 *  its longest chains. Fitted to calls of 5,000 to 250,000 pairs in either form (DNA profiles / compared text, halves ->
 *  quarters): 45,000 pairs of 30 x 600 500 -> 1,170 us / 505 -> 538, 250,000 1,680 -> 1,700 / 1,750 -> 1,590; 20,000 pairs
 *  of 100-300 on either side 407 -> 573 / 390 -> 400, 45,000 753 -> 672 / 722 -> 607; 65,536 of 40-200 476 -> 523 / 448 ->
 *  415, 100,000 640 -> 576 / 608 -> 543; 150,000 of 16-128 374 -> 402 / 370 -> 389. */
__host__ __device__ inline float short_fine_rows(float rows, float columns, bool profile) {
    bool const uneven = columns > 1.3f * rows;
    if (!profile) return 6.2e6f - 1.3e4f * rows;
    if (uneven) return rows < 56.0f ? 1.5e7f : 1.0e7f - 2.7e4f * rows;
    return 8.0e6f - 1.2e4f * rows;
}
static_assert(bin_short_begin_k + short_shapes_k * short_m_classes_k <= bin_keys_k, "bin layout exceeds the key space");
constexpr int bin_myers_chain_k = bin_short_begin_k + short_shapes_k * short_m_classes_k; // 2028
/** Rows of a segment of one shape, on the host and on the device. */
__host__ __device__ constexpr int short_segment_rows(int shape) {
    return shape == 0 ? 16 : (16 << ((shape - 1) / 4)) / 4 * (5 + (shape - 1) % 4);
}
static_assert(short_segment_rows(short_shapes_k - 1) == short_max_rows_k, "the last shape holds the longest short pairs");

__host__ __device__ inline int floor_log2_u64(std::uint64_t x) {
#ifdef __CUDA_ARCH__
    return x ? 63 - __clzll((long long)x) : 0;
#else
    return x ? 63 - __builtin_clzll(x) : 0;
#endif
}

/** Bin of a short pair of n rows (at most 448) and m >= n columns, its rows cut in quarters of an octave when `fine`, else
 *  in halves. Classes of 16 columns over the rows of the next smaller shape, then octaves of that excess, which has 64 bits:
 *  a local pair's text may have 2^31 symbols and more. */
__host__ __device__ inline int short_bin(std::uint64_t n, std::uint64_t m, bool fine) {
    int const octave = n <= 16 ? 0 : floor_log2_u64(n - 1) - 4;
    int quarter = n <= 16 ? -1 : int((n - 1) >> (octave + 2)) - 4;
    if (!fine) quarter |= 1;
    std::uint64_t const smaller = n <= 16 ? 0 : (4u << octave) * (fine ? 4u + quarter : 3u + quarter);
    std::uint64_t const excess = m - smaller;
    int const octaves = floor_log2_u64(excess) - 8;
    int const m_class = excess < 320 ? int(excess / 16) : 20 + (octaves < 6 ? octaves : 6);
    return bin_short_begin_k + (1 + 4 * octave + quarter) * short_m_classes_k + (short_m_classes_k - 1 - m_class);
}

static_assert(bin_myers_chain_k < bin_keys_k, "bin layout exceeds the key space");
constexpr int near_min_words_k = 5; // patterns of the thread route that the near-diagonal kernel tries
constexpr std::uint32_t near_samples_k = 128; // pairs sampled per call
constexpr int near_unrelated_edits_k = 6;     // fewest edits in 16 rows at either end of a pair that counts as unrelated
constexpr std::uint64_t near_large_pairs_k = 100000; // pairs from which the trial's left-over does not cost its chain
constexpr std::uint32_t near_trial_k = 4096; // pairs tried near the diagonal before a batch may be found unrelated
constexpr std::uint32_t myers_chain_max_rows_k = 1u << 20; // longest pattern a chain of warps takes

/** Which pairs a call scores. */
enum pair_mode_t : int {
    mode_pairwise_k = 0,  // (i, i)
    mode_cross_k = 1,     // (q, c) for all q, c
    mode_symmetric_k = 2, // (q, c) for c <= q, mirrored on output
};

/** A tape as the kernels see it: `base + offsets[i]` is the start of string i, which ends where string i + 1 starts, or
 *  after `lengths[i]` symbols where there are lengths (transcoded UTF-8: codes at the positions of the bytes). */
struct tape_t {
    std::uint8_t const *base;
    void const *offsets;
    std::uint64_t count;
    int offset_bits; // 32 or 64
    std::uint64_t const *lengths;
};

/** Everything the planning kernels need. */
struct plan_args_t {
    tape_t queries, candidates;
    int mode;
    std::uint64_t pairs;
    std::uint64_t candidates_count; // columns of the cross product
    int kind, affine;
    int open, extend, match, mismatch;
    int unit_levenshtein;   // 0/1/1/1 Levenshtein: bit-parallel route
    int magnitude;          // max |cost| over substitution and gap costs, at least 1
    int local_gain;         // local scores with non-positive gaps: max(0, largest substitution cost); else -1
    int steps_beyond_span;  // 1 linear, 3 affine (serial.hpp:126-140)
    int force_route;        // -1: normal planning; otherwise one bin per route, input order (the plain form)
    int wide;               // UTF-8 calls over more than 256 code points: the tapes hold 16-bit codes, offsets in codes
    int packed_allowed;     // 1 if the 16x2 route may hold the substitution costs in int8 profiles
    int dense;              // dense-table engine: its profile holds the batch's bytes, at most 32 of them
    batch_alphabet_t const *alphabet; // Levenshtein: the batch alphabet, read on the device (may be null)
    // Tuning by length class k = floor(log2(shorter side)), 15 for everything longer.
    std::uint8_t packed_rows[16];     // 0: per-pair step-cost model; else rows per lane 4, 8, 12, 16
    std::uint8_t cell_bits[16];       // 0: narrowest safe; 32: never 16-bit cells; 64: 64-bit cells
    std::uint32_t band_min_rows;      // shorter sides above this take the band (pairs on 32-bit cells)
    std::uint32_t band_min_rows_packed; // the same for pairs that fit 16-bit cells
    std::uint16_t packed_step_cost[4];  // relative cost of one lane step with 4, 8, 12, 16 rows per lane
    std::uint32_t band_min_rows_compare; // the same for compare-mode Levenshtein pairs (no profile)
    std::uint32_t short_max_rows;        // 16x2 pairs whose shorter side is at most this take the short route
    int short_fine;                      // 1: quarter octaves of rows, where the profile has few classes
    int classes;                         // profile classes of the engine's table (not read for Levenshtein or dense)
    std::uint32_t near_sample_stride;    // unit-cost calls: every so many pairs one is sampled for likeness (0: none)
    int near_long;                       // 1: pairs enough for the nine-word window of patterns past the thread route
};

/** What the ends of sampled pairs say about trying a call's pairs near their diagonal first (myers_near.cuh). */
struct near_sample_t {
    std::uint32_t sampled;   // pairs sampled that the near-diagonal kernels could take
    std::uint32_t unrelated; // unrelated, or of lengths too different
    std::uint32_t alike;     // at a distance well inside the kernels' limits
    std::uint32_t edits;     // of all related ones' 32 rows at both ends
};

/**
 *  Whether @p pairs with patterns of up to @p longest rows should be tried near their diagonal (`half` blocks either side)
 *  before the full kernels score what is left. A pair found saves a third of its work or more, but what is left over starts
 *  only when all have been tried, so a few failures cost a call of less than some waves of threads a whole full kernel's
 *  chain. Such a call has to have hardly an unrelated pair, and its longest pairs at the sampled rate of edits have to stay
 *  inside the limit; a larger one needs a third of its pairs alike and less than half unrelated. Against never trying: 20,000
 *  DNA reads of 100-300 at 8-18 % substitutions 1.17-1.25x, at 22 % 0.80x, half of them unrelated 0.77x; 5,000 of
 *  1,000-4,000 with a tenth unrelated 0.76x, at 8 % 1.05x, at 4 % 2.6x; 200,000 of 100-300 at 26 % 1.18x, with 35 %
 *  unrelated 1.08x, with half 0.98x, with 65 % 0.90x.
 */
inline bool near_pays(near_sample_t const &sample, std::uint64_t pairs, std::uint32_t longest, int half) {
    if (pairs >= near_large_pairs_k)
        return sample.alike * 3 > sample.sampled && sample.unrelated * 20 <= sample.sampled * 9;
    if (!sample.alike || sample.unrelated * 32 > sample.sampled) return false;
    float const edits = (float)sample.edits / (32.0f * (float)(sample.sampled - sample.unrelated)) * (float)longest;
    float const room = 64.0f * (float)half - edits;
    return room > 0 && edits * (2.8f * 2.8f) <= room * room; // 2.8 standard deviations
}

/** Per-bin counters the planner fills. */
struct plan_bins_t {
    std::uint32_t count[bin_keys_k];
    std::uint32_t begin[bin_keys_k];
    std::uint32_t fill[bin_keys_k];
    std::uint32_t cursor[bin_keys_k];
    std::uint32_t max_cols;
    std::uint32_t error_flags;
    std::uint64_t cells;
    std::uint64_t scheduled;
    std::uint32_t max_myers_rows;      // longest pattern on the thread-per-pair bit-parallel route
    std::uint32_t max_myers_warp_rows; // longest pattern on the warp-per-pair bit-parallel route
    std::uint32_t max_chain_rows;      // longest pattern on the chained bit-parallel route
    std::uint32_t near_tried, near_failed; // pairs the near-diagonal kernel has tried, and those it had to list
    near_sample_t near;                     // the planner's look at the pairs' likeness
    std::uint32_t short_fine;              // whether short pairs are cut in quarter octaves (`short_fine_rows`)
    std::uint32_t listed[32];              // pairs it listed per class of full kernel (words; 16 + words per lane)
};

} // namespace szs_gb300
