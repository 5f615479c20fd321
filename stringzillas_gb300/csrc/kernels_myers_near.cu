/**
 *  @file kernels_myers_near.cu
 *  @brief Instantiations of the near-diagonal bit-parallel kernel.
 */
#include "launchers.h"
#include "myers_near.cuh"

namespace szs_gb300 {

template <int half_, int mode_>
static cudaError_t near_launch(pair_task_t const *tasks, plan_bins_t *bins, int key_begin, int key_end,
                               batch_alphabet_t const *alphabet, std::int64_t *results, std::uint32_t *list, int ctas,
                               cudaStream_t stream) {
    myers_near_kernel<half_, mode_><<<ctas, near_threads_k, near_shared_bytes(half_, mode_), stream>>>(
        tasks, bins, key_begin, key_end, alphabet, results, list);
    return cudaGetLastError();
}

int myers_near_threads() { return near_threads_k; }

cudaError_t launch_myers_near(int half, int planes, pair_task_t const *tasks, plan_bins_t *bins, int key_begin,
                              int key_end, batch_alphabet_t const *alphabet, std::int64_t *results,
                              std::uint32_t *list, int ctas, cudaStream_t stream) {
    int const mode = planes == 2 ? near_dna_k : (planes == 16 ? near_wide_k : near_bytes_k);
    if (half == 1 && mode == near_dna_k)
        return near_launch<1, near_dna_k>(tasks, bins, key_begin, key_end, alphabet, results, list, ctas, stream);
    if (half == 1 && mode == near_bytes_k)
        return near_launch<1, near_bytes_k>(tasks, bins, key_begin, key_end, alphabet, results, list, ctas, stream);
    if (half == 1 && mode == near_wide_k)
        return near_launch<1, near_wide_k>(tasks, bins, key_begin, key_end, alphabet, results, list, ctas, stream);
    if (half == 4 && mode == near_dna_k)
        return near_launch<4, near_dna_k>(tasks, bins, key_begin, key_end, alphabet, results, list, ctas, stream);
    return cudaErrorInvalidValue;
}

} // namespace szs_gb300
