/**
 *  @file kernels_short.cu
 *  @brief Instantiations and launcher of the segmented 16x2 kernel for short pairs (dp_short.cuh) for every cost
 *         family, profile and compare modes. Segment shape 0 holds 16 rows; the octave above 16 << k has four shapes,
 *         1 + 4 k + q, of 5/4, 6/4, 7/4 and 8/4 times its start. With few classes or in compare mode they are 2^k lanes
 *         x 20, 24 and 28 rows and 2^(k + 1) lanes x 16 rows; profiles over many classes, whose segments together stay
 *         near 32 x 8 rows per pair and warp in shared memory, have the 6/4 and 8/4 shapes with 2^(k + 1) lanes x 12
 *         and 2^(k + 2) lanes x 8 rows.
 *
 *  Compiled six times, with `SZS_SHORT_ROWS` 8, 12, 16, 20, 24 or 28, so the families build in parallel.
 */
#include "dp_short.cuh"
#include "launchers.h"

#ifndef SZS_SHORT_ROWS
#error "compile with -DSZS_SHORT_ROWS=<8|12|16|20|24|28>"
#endif

namespace szs_gb300 {

namespace {

template <int kind_, bool affine_, int lanes_, int rows_, int compare_>
dp_launch_shape_t short_shape_of(int classes, int warps) {
    using policy_t = short_policy_t<kind_, affine_, lanes_, rows_, compare_>;
    dp_launch_shape_t shape;
    shape.threads_per_cta = warps * 32;
    shape.warps_per_cta = warps;
    shape.rows_per_lane = rows_;
    shape.shared_bytes = short_shared_bytes<policy_t>(warps, classes);
    auto kernel = dp16_short_kernel<policy_t>;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, shape.shared_bytes);
    int blocks = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kernel, shape.threads_per_cta, shape.shared_bytes) !=
        cudaSuccess)
        blocks = 0;
    shape.ctas_per_sm = blocks;
    return shape;
}

template <int kind_, bool affine_, int lanes_, int rows_, int compare_>
cudaError_t short_launch_of(int key_begin, int key_end, pair_task_t const *tasks, plan_bins_t *bins,
                            score_costs_t const &costs, std::int64_t *results, int ctas, int warps,
                            cudaStream_t stream) {
    using policy_t = short_policy_t<kind_, affine_, lanes_, rows_, compare_>;
    int const shared = short_shared_bytes<policy_t>(warps, costs.classes);
    auto kernel = dp16_short_kernel<policy_t>;
    cudaError_t status = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, shared);
    if (status != cudaSuccess) return status;
    kernel<<<ctas, warps * 32, shared, stream>>>(tasks, bins, key_begin, key_end, costs, results);
    return cudaGetLastError();
}

// Lanes per segment: 1 to 16, but not one lane of 8 or 12 rows.
#if SZS_SHORT_ROWS < 16
#define SZS_SHORT_LANES_1(call_, kind_, affine_, compare_, ...)
#else
#define SZS_SHORT_LANES_1(call_, kind_, affine_, compare_, ...)                                                      \
    case 1: return call_<kind_, affine_, 1, SZS_SHORT_ROWS, compare_>(__VA_ARGS__);
#endif
#define SZS_SHORT_LANES(call_, kind_, affine_, compare_, ...)                                                        \
    switch (lanes) {                                                                                                 \
    SZS_SHORT_LANES_1(call_, kind_, affine_, compare_, __VA_ARGS__)                                                  \
    case 2: return call_<kind_, affine_, 2, SZS_SHORT_ROWS, compare_>(__VA_ARGS__);                                  \
    case 4: return call_<kind_, affine_, 4, SZS_SHORT_ROWS, compare_>(__VA_ARGS__);                                  \
    case 8: return call_<kind_, affine_, 8, SZS_SHORT_ROWS, compare_>(__VA_ARGS__);                                  \
    case 16: return call_<kind_, affine_, 16, SZS_SHORT_ROWS, compare_>(__VA_ARGS__);                                \
    default: break;                                                                                                  \
    }

#if SZS_SHORT_ROWS == 8
#define SZS_SHORT_COMPARE(call_, ...) break; // profiles over many classes only
#else
#define SZS_SHORT_COMPARE(call_, ...)                                                                                \
    if (kind != kind_levenshtein_k) break;                                                                           \
    switch ((affine ? 2 : 0) + (compare == compare_multiply_k ? 1 : 0)) {                                            \
    case 0: SZS_SHORT_LANES(call_, kind_levenshtein_k, false, compare_select_k, __VA_ARGS__) break;                  \
    case 1: SZS_SHORT_LANES(call_, kind_levenshtein_k, false, compare_multiply_k, __VA_ARGS__) break;                \
    case 2: SZS_SHORT_LANES(call_, kind_levenshtein_k, true, compare_select_k, __VA_ARGS__) break;                   \
    default: SZS_SHORT_LANES(call_, kind_levenshtein_k, true, compare_multiply_k, __VA_ARGS__) break;                \
    }                                                                                                                \
    break;
#endif

#if SZS_SHORT_ROWS > 16
#define SZS_SHORT_ROW_MAXIMA(call_, ...) break; // up to 128 rows in halves of octaves only
#else
#define SZS_SHORT_ROW_MAXIMA(call_, ...)                                                                             \
    if (kind != kind_smith_waterman_k) break;                                                                        \
    if (affine) SZS_SHORT_LANES(call_, kind_smith_waterman_k, true, short_row_maxima_k, __VA_ARGS__)                 \
    else SZS_SHORT_LANES(call_, kind_smith_waterman_k, false, short_row_maxima_k, __VA_ARGS__)                       \
    break;
#endif

#define SZS_SHORT_DISPATCH(call_, ...)                                                                               \
    if (compare == short_row_maxima_k) {                                                                             \
        SZS_SHORT_ROW_MAXIMA(call_, __VA_ARGS__)                                                                     \
    }                                                                                                                \
    if (compare != compare_none_k) {                                                                                 \
        SZS_SHORT_COMPARE(call_, __VA_ARGS__)                                                                        \
    }                                                                                                                \
    switch (kind * 2 + (affine ? 1 : 0)) {                                                                           \
    case 0: SZS_SHORT_LANES(call_, kind_levenshtein_k, false, compare_none_k, __VA_ARGS__) break;                    \
    case 1: SZS_SHORT_LANES(call_, kind_levenshtein_k, true, compare_none_k, __VA_ARGS__) break;                     \
    case 2: SZS_SHORT_LANES(call_, kind_needleman_wunsch_k, false, compare_none_k, __VA_ARGS__) break;               \
    case 3: SZS_SHORT_LANES(call_, kind_needleman_wunsch_k, true, compare_none_k, __VA_ARGS__) break;                \
    case 4: SZS_SHORT_LANES(call_, kind_smith_waterman_k, false, compare_none_k, __VA_ARGS__) break;                 \
    case 5: SZS_SHORT_LANES(call_, kind_smith_waterman_k, true, compare_none_k, __VA_ARGS__) break;                  \
    default: break;                                                                                                  \
    }

} // namespace

#define SZS_CONCAT_(a, b) a##b
#define SZS_CONCAT(a, b) SZS_CONCAT_(a, b)

dp_launch_shape_t SZS_CONCAT(short_shape_rows, SZS_SHORT_ROWS)(int kind, bool affine, int lanes, int classes,
                                                               int warps, int compare) {
    if (warps >= 1 && warps <= 4) do {
            SZS_SHORT_DISPATCH(short_shape_of, classes, warps)
        } while (false);
    return dp_launch_shape_t {0, 0, 0, 0, 0};
}

cudaError_t SZS_CONCAT(launch_short_rows, SZS_SHORT_ROWS)(int kind, bool affine, int lanes, int key_begin,
                                                           int key_end, pair_task_t const *tasks, plan_bins_t *bins,
                                                           score_costs_t const &costs, std::int64_t *results,
                                                           int ctas, int warps, cudaStream_t stream, int compare) {
    if (warps >= 1 && warps <= 4) do {
            SZS_SHORT_DISPATCH(short_launch_of, key_begin, key_end, tasks, bins, costs, results, ctas, warps, stream)
        } while (false);
    return cudaErrorInvalidValue;
}

#if SZS_SHORT_ROWS == 16

#define SZS_SHORT_DECLARE(rows_)                                                                                     \
    dp_launch_shape_t short_shape_rows##rows_(int kind, bool affine, int lanes, int classes, int warps, int compare); \
    cudaError_t launch_short_rows##rows_(int kind, bool affine, int lanes, int key_begin, int key_end,               \
                                         pair_task_t const *tasks, plan_bins_t *bins, score_costs_t const &costs,    \
                                         std::int64_t *results, int ctas, int warps, cudaStream_t stream,            \
                                         int compare);
SZS_SHORT_DECLARE(8)
SZS_SHORT_DECLARE(12)
SZS_SHORT_DECLARE(20)
SZS_SHORT_DECLARE(24)
SZS_SHORT_DECLARE(28)

int short_rows_for(int classes, int compare, int shape, std::uint64_t pairs, int sm_count) {
    bool const row_maxima = compare == short_row_maxima_k;
    bool const few = (compare != compare_none_k && !row_maxima) || classes <= short_few_classes_k;
    int const quarter = shape == 0 ? 3 : (shape - 1) % 4;
    if (quarter == 3) return few ? 16 : 8;
    if (!few || row_maxima) return 12;
    // The 6/4 shapes up to 16 lanes have a second form of half the rows in twice the lanes, whose steps are half as
    // long: where the pairs leave warp slots free, a warp's own chain of steps is what takes the time.
    int const lanes = short_segment_rows(shape) / 24;
    std::uint64_t const warps = pairs / (64u / lanes);
    return quarter == 1 && lanes <= 8 && warps < 64u * (std::uint64_t)sm_count ? 12 : 20 + 4 * quarter;
}

dp_launch_shape_t short_shape(int kind, bool affine, int shape, int rows, int classes, int warps, int compare) {
    int const lanes = short_segment_rows(shape) / rows;
    switch (rows) {
    case 8: return short_shape_rows8(kind, affine, lanes, classes, warps, compare);
    case 12: return short_shape_rows12(kind, affine, lanes, classes, warps, compare);
    case 16: return short_shape_rows16(kind, affine, lanes, classes, warps, compare);
    case 20: return short_shape_rows20(kind, affine, lanes, classes, warps, compare);
    case 24: return short_shape_rows24(kind, affine, lanes, classes, warps, compare);
    default: return short_shape_rows28(kind, affine, lanes, classes, warps, compare);
    }
}

cudaError_t launch_short(int kind, bool affine, int shape, int rows, int key_begin, int key_end,
                         pair_task_t const *tasks, plan_bins_t *bins, score_costs_t const &costs,
                         std::int64_t *results, int ctas, int warps, cudaStream_t stream, int compare) {
    int const lanes = short_segment_rows(shape) / rows;
    auto const launch = rows == 8    ? launch_short_rows8
                        : rows == 12 ? launch_short_rows12
                        : rows == 16 ? launch_short_rows16
                        : rows == 20 ? launch_short_rows20
                        : rows == 24 ? launch_short_rows24
                                     : launch_short_rows28;
    return launch(kind, affine, lanes, key_begin, key_end, tasks, bins, costs, results, ctas, warps, stream, compare);
}

#endif

} // namespace szs_gb300
