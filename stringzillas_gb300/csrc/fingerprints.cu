/**
 *  @file fingerprints.cu
 *  @brief Min-Hash fingerprints (the reference's `szs_fingerprints_*`): per text and dimension, the minimum
 *         rolling hash over all windows of the dimension's width, and how often that minimum occurs.
 *
 *  Dimension d rolls a Rabin-Karp hash over bytes + 1 modulo m_d with multiplier a_d, both drawn from `splitmix64`
 *  streams of `seed + d` (include/stringzillas/fingerprints/serial.hpp:33-41, :426-432). The reference evaluates it
 *  in double precision with Barrett reductions (:1040-1050) that are exact on these magnitudes, so exact integer
 *  arithmetic gives the same residues. Each step here is one reduction of `state * a + byte_in + 1 + D *
 *  (byte_out + 1)` with D = -a^w mod m, the reference's two reductions (drop the outgoing byte, append the incoming
 *  one) folded into one.
 *
 *  Magnitudes: 2^42 < m < 2^43 and a < 640. The rolling state is kept in [0, 2m) rather than [0, m): any
 *  representative continues the recurrence, and the conditional subtraction that would make it canonical is only
 *  paid where the running minimum needs it. Then x < 2m * a + 256 * D + 256 < 2^54, every product is a 32 x 64-bit
 *  one (two multiply-adds), and the quotient is estimated from the top 32 bits of x: with t = x >> 22 and
 *  mu = floor(2^74 / m), floor(t * mu / 2^52) is q or q - 1 (the dropped low bits and mu's truncation each cost
 *  less than 2^-20 of a unit), so x - estimate * m lies in [0, 2m) again.
 *
 *  The running minimum is over canonical values c = state or state - m. A window can only reach it when the high
 *  words pass `state_hi <= min_hi || state_hi - m_hi <= min_hi + 1` (a borrow can lower state - m's high word by one),
 *  a 32-bit test that fails for nearly every window of a long text; the exact comparison runs behind it.
 *
 *  Two kernels share this arithmetic. Windows of up to 32 bytes (`fingerprints_tensor_kernel`): a window's hash as a
 *  fraction of its modulus is a dot product of its bytes with w fixed weights, so tensor cores evaluate it for every
 *  window and dimension to 22 bits, and only windows that could be the minimum are hashed exactly. Wider windows
 *  (`fingerprints_kernel`): one warp rolls 32 consecutive dimensions of one text exactly; the lanes read the same byte
 *  stream and write 32 adjacent outputs.
 */
#include "launchers.h"

#include <algorithm>
#include <cmath>
#include <cstdlib>

namespace szs_gb300 {

namespace {

constexpr int tensor_width_k = fingerprint_tensor_width_k;   // widest window the tensor-core kernel takes
constexpr int tensor_tiles_k = 8;                            // tiles of 8 dimensions per warp
constexpr int tensor_dims_k = fingerprint_group_k;           // 64 dimensions per warp
static_assert(tensor_dims_k == 8 * tensor_tiles_k, "a warp's dimensions are whole tiles");
constexpr int tensor_chunk_k = 256;                          // window starts per staged chunk
constexpr int tensor_staged_k = tensor_chunk_k + 2 * tensor_width_k; // byte pairs staged per chunk
constexpr std::uint32_t tensor_list_k = 512;                 // candidate windows a chunk may list
constexpr int tensor_warps_k = 4;                            // warps per CTA, each on its own text and dimensions

/** A representative in [0, 2m) of x mod m, for x < 2^54 (see the file comment). */
__device__ __forceinline__ std::uint64_t reduce(std::uint64_t x, std::uint64_t modulo, std::uint32_t mu) {
    std::uint32_t const top = (std::uint32_t)(x >> 22);
    std::uint32_t const quotient = __umulhi(top, mu) >> 20;
    return x - (std::uint64_t)quotient * modulo;
}

__device__ __forceinline__ std::uint64_t canonical(std::uint64_t r, std::uint64_t modulo) {
    return r >= modulo ? r - modulo : r;
}

__device__ __forceinline__ std::uint64_t text_offset(tape_t const &tape, std::uint64_t i) {
    return tape.offset_bits == 32 ? static_cast<std::uint32_t const *>(tape.offsets)[i]
                                  : static_cast<std::uint64_t const *>(tape.offsets)[i];
}

/** Two bytes at once: a representative in [0, 2m) of x mod m for x < 2^62, the quotient (below 2^20) from x's top 32
 *  bits: with t = x >> 30, floor(t * mu / 2^44) is q or q - 1 (both truncations cost less than 2^-11 of a unit). */
__device__ __forceinline__ std::uint64_t reduce_wide(std::uint64_t x, std::uint64_t modulo, std::uint32_t mu) {
    std::uint32_t const top = (std::uint32_t)(x >> 30);
    std::uint32_t const quotient = __umulhi(top, mu) >> 12;
    return x - (std::uint64_t)quotient * modulo;
}

/** The canonical hash of the `width` bytes at `window`, two bytes per reduction: state < 2m < 2^43.1 and a^2 < 2^18.7
 *  keep every intermediate below 2^62. */
__device__ __forceinline__ std::uint64_t window_hash(std::uint8_t const *window, std::uint32_t width,
                                                     std::uint32_t multiplier, std::uint64_t modulo,
                                                     std::uint32_t mu) {
    std::uint32_t const square = multiplier * multiplier;
    std::uint64_t state = 0;
    std::uint32_t i = 0;
    if (width & 1u) state = window[i++] + 1u;
    for (; i < width; i += 2) {
        std::uint32_t const two = (window[i] + 1u) * multiplier + window[i + 1] + 1u;
        state = reduce_wide(state * square + two, modulo, mu);
    }
    return canonical(state, modulo);
}

/** One dimension's rolling hash over consecutive windows, with the running minimum of its canonical values and its
 *  number of occurrences (all ones and 0 before any window), without branches: in repeats some lane of a warp counts at
 *  nearly every step. */
struct rolling_t {
    std::uint64_t state, minimum, modulo, discard;
    std::uint32_t occurrences, multiplier, mu, width;

    __device__ __forceinline__ void open(fingerprint_dim_t const &p, std::uint64_t minimum_, std::uint32_t occurrences_) {
        modulo = p.modulo, discard = p.discard, multiplier = p.multiplier, mu = p.mu, width = p.width;
        minimum = minimum_, occurrences = occurrences_;
    }
    __device__ __forceinline__ void take() {
        std::uint64_t const value = canonical(state, modulo);
        bool const lower = value < minimum;
        occurrences = (lower ? 0u : occurrences) + (value <= minimum ? 1u : 0u);
        minimum = lower ? value : minimum;
    }
    /** The window starting at `window`, from its bytes alone. */
    __device__ __forceinline__ void first(std::uint8_t const *window) {
        state = window_hash(window, width, multiplier, modulo, mu);
        take();
    }
    /** The next window, dropping byte `out` and taking byte `in`. */
    __device__ __forceinline__ void next(std::uint32_t out, std::uint32_t in) {
        // in + 1 + D * (out + 1) = in + D * out + (D + 1)
        state = reduce(state * multiplier + discard * out + (discard + 1u + in), modulo, mu);
        take();
    }
};

/** Whether a text has fewer windows (of its group's widest dimension) than pay for bounding the minimum by tensor-core tiles
 *  before its candidates are listed: it is rolled exactly. */
__device__ __forceinline__ bool rolls(std::uint64_t length, std::uint32_t widest, std::uint32_t windows_min) {
    return length < widest + (windows_min - 1u);
}

/** The fewest windows of a tensor-core text. The tensor kernel's chain per text is longer at the start than a short text's
 *  rolled one, so calls that leave warp slots free roll longer texts than those that fill them. Rolled / tensor: 1 to 64
 *  texts of 200 bytes at 64 to 1,024 dimensions 46 / 49 us, of 300 56 / 53; 1,000 of 100-200 at 64 dimensions 53 / 73; 250 of
 *  150 at 1,024 81 / 92, of 200 102 / 83 (but 1,000 of 100-200 at 256, of which a quarter pass the line, 105 / 130); 4,000 of
 *  150 at 1,024 815 / 688. */
std::uint32_t tensor_windows_min(std::uint64_t items, int sm_count) {
    return items <= 12ull * sm_count ? 224 : items <= 48ull * sm_count ? 160 : 128;
}

/** What one warp of the tensor-core kernel keeps in shared memory. */
struct __align__(16) tensor_warp_t {
    unsigned long long minimum[tensor_dims_k]; // exact minimum so far (all ones: no window yet)
    std::uint32_t occurrences[tensor_dims_k];
    std::uint32_t width[tensor_dims_k];
    std::uint32_t margin[tensor_dims_k];
    std::uint32_t mu[tensor_dims_k], shift[tensor_dims_k];
    std::uint32_t limit[tensor_dims_k];        // largest estimate of a window that could still be the minimum
    std::uint32_t pairs[tensor_staged_k];      // halves of bytes (p, p + 1) of the chunk, for every p
    std::uint16_t list[tensor_list_k];         // candidates of the chunk: dimension << 8 | window
    std::uint32_t listed;
};

/** d = a (16 windows x 16 bytes) * b (16 weights x 8 dimensions) + c, halves into single precision. */
__device__ __forceinline__ void mma_tile(float (&d)[4], std::uint32_t a0, std::uint32_t a1, std::uint32_t a2,
                                         std::uint32_t a3, std::uint32_t b0, std::uint32_t b1, float c0, float c1,
                                         float c2, float c3) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%10, %11, %12, %13};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(c0), "f"(c1), "f"(c2), "f"(c3));
}

/**
 *  Min-Hash over windows of at most 16 x `steps_` bytes: one warp per text and 64 dimensions, on tensor cores.
 *
 *  hash / m = sum over the window's bytes of c_i * (a^(w-1-i) mod m) / m, modulo 1, with c = byte + 1. Each weight is
 *  rounded to 22 fractional bits and split into two signed 11-bit digits, and c is centred (c - 128, the constant
 *  128 * sum of weights kept apart), so both digit sums are integers of at most 32 * 128 * 1024 = 2^22 in magnitude:
 *  started from 1.5 * 2^23 they stay single-precision integers in [2^23, 2^24], exact in any order of summation, whose
 *  bit patterns are a constant plus the integer. Hashes of windows too short to wrap around the modulus fill a small
 *  part of its range: their weights are scaled up by `2^shift`. The constant vanishes modulo 2^32 under the digits' shifts, so
 *  `bits_hi << 21 + bits_lo << 10 + offset` is the fraction in units of 2^-32, off by at most the dimension's `margin`
 *  (128 * sum of the weights' rounding errors, computed per dimension on the host).
 *
 *  The windows' Toeplitz matrix costs one shared-memory word per lane and 8 windows: entry (p, i) is byte p + i, so
 *  the fragments of neighbouring tiles and halves coincide. A window is a candidate when its estimate (biased up by
 *  the margin, so never wrapped below 0) is at most `limit`, an upper bound of what any minimal window's estimate can
 *  be; candidates are listed, hashed exactly 32 at a time after each chunk of 256 windows, and tighten the limits. So
 *  the results are those of exact hashes alone. A chunk with more candidates than the list holds (a run of one byte)
 *  is rolled exactly instead.
 *
 *  16,384 texts of 1,000-3,000 bytes at 1,024 dimensions: 40.4 ms rolled, 15.9 ms here (2.1 T byte-dimensions/s; 2.5 T
 *  for windows of up to 16 bytes, 1.4 T for wider ones).
 *
 *  Bound: issue of the estimates' epilogue (two multiply-adds and a compare per window and dimension, half a tensor
 *  instruction) rather than the tensor pipe, which is why the register-accumulator form is used: accumulators in
 *  tensor memory would add a load of each to the same epilogue.
 */
template <int steps_>
__global__ void __launch_bounds__(32 * tensor_warps_k, steps_ == 1 ? 4 : 3)
    fingerprints_tensor_kernel(tape_t const texts, fingerprint_dim_t const *__restrict__ params,
                               fingerprint_weights_t const *__restrict__ digits, std::uint32_t const dimensions,
                               fingerprint_group_t const *__restrict__ groups, std::uint32_t const groups_count,
                               std::uint32_t const windows_min, std::uint32_t *__restrict__ hashes,
                               std::uint64_t const hashes_stride, std::uint32_t *__restrict__ counts,
                               std::uint64_t const counts_stride) {
    extern __shared__ __align__(16) unsigned char tensor_s[];
    int const lane = threadIdx.x & 31, row = lane >> 2, column = (lane & 3) * 2;
    tensor_warp_t &own = reinterpret_cast<tensor_warp_t *>(tensor_s)[threadIdx.x / 32];
    std::uint64_t const warp = (std::uint64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    std::uint64_t const slots = (std::uint64_t)gridDim.x * (blockDim.x / 32) / groups_count; // warps per group
    asm volatile("griddepcontrol.launch_dependents;"); // the kernels of a call write different outputs
    if (warp >= slots * groups_count) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        return;
    }
    fingerprint_group_t const group = groups[warp % groups_count];
    std::uint32_t const first_dim = group.index * tensor_dims_k, widest = group.widest;
    constexpr float bias = 12582912.0f; // 1.5 * 2^23

    // The warp's next text that is not the rolling kernel's, found 32 at a time.
    auto seek = [&](std::uint64_t text) {
        for (; text < texts.count; text += 32 * slots) {
            std::uint64_t const candidate = text + lane * slots;
            bool const mine = candidate < texts.count &&
                              !rolls(text_offset(texts, candidate + 1) - text_offset(texts, candidate), widest,
                                     windows_min);
            if (std::uint32_t const found = __ballot_sync(0xFFFFFFFFu, mine)) return text + (__ffs(found) - 1) * slots;
        }
        return texts.count;
    };
    std::uint64_t const first_text = seek(warp / groups_count);
    if (first_text >= texts.count) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        return;
    }

    // The group's weights as fragments, and each lane's dimensions (8 tile + column, + 1).
    std::uint32_t weights[tensor_tiles_k][2][steps_][2];
    std::uint32_t offset[tensor_tiles_k][2];
    for (int k = lane; k < tensor_dims_k; k += 32) {
        fingerprint_dim_t const &p = params[min(first_dim + k, dimensions - 1)];
        own.width[k] = p.width, own.margin[k] = p.margin, own.mu[k] = p.mu, own.shift[k] = p.shift;
    }
    std::uint32_t narrowest = 0xFFFFFFFFu;
    __syncwarp();
    for (int k = lane; k < tensor_dims_k; k += 32) narrowest = min(narrowest, own.width[k]);
    narrowest = __reduce_min_sync(0xFFFFFFFFu, narrowest);
#pragma unroll
    for (int tile = 0; tile < tensor_tiles_k; ++tile) {
        fingerprint_weights_t const &p = digits[min(first_dim + 8 * tile + row, dimensions - 1)];
#pragma unroll
        for (int digit = 0; digit < 2; ++digit)
#pragma unroll
            for (int step = 0; step < steps_; ++step)
#pragma unroll
                for (int half = 0; half < 2; ++half)
                    weights[tile][digit][step][half] =
                        *reinterpret_cast<std::uint32_t const *>(&p.digits[digit][16 * step + 8 * half + column]);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            fingerprint_dim_t const &q = params[min(first_dim + 8 * tile + column + j, dimensions - 1)];
            offset[tile][j] = q.offset + q.margin;
        }
    }

    for (std::uint64_t text = first_text; text < texts.count; text = seek(text + slots)) {
        std::uint64_t const start = text_offset(texts, text);
        std::uint64_t const length = text_offset(texts, text + 1) - start;
        std::uint8_t const *bytes = texts.base + start;
        __syncwarp();
        for (int k = lane; k < tensor_dims_k; k += 32)
            own.minimum[k] = ~0ull, own.occurrences[k] = 0, own.limit[k] = 0xFFFFFFFFu;
        std::uint32_t limit[tensor_tiles_k][2];
#pragma unroll
        for (int tile = 0; tile < tensor_tiles_k; ++tile) limit[tile][0] = limit[tile][1] = 0xFFFFFFFFu;
        std::uint64_t const windows = length - narrowest + 1;
        for (std::uint64_t base = 0; base < windows; base += tensor_chunk_k) {
            std::uint32_t const here = (std::uint32_t)min((std::uint64_t)tensor_chunk_k, windows - base);
            {
                __syncwarp();
                // Positions past the text stage as zeros: their windows are never counted.
                std::uint8_t const *ahead = bytes + base + lane;
                std::uint32_t const left = (std::uint32_t)min(length - base, (std::uint64_t)tensor_staged_k + 1);
#pragma unroll
                for (std::uint32_t i = 0; i < tensor_staged_k; i += 32) {
                    std::uint32_t const p = i + lane;
                    std::uint32_t const low = p < left ? ahead[i] : 127u, high = p + 1 < left ? ahead[i + 1] : 127u;
                    // 0x6400 | x is the half 1024 + x; minus 1,151 leaves x + 1 - 128.
                    std::uint32_t const packed = 0x64006400u | low | high << 16;
                    std::uint32_t centred;
                    asm("sub.f16x2 %0, %1, %2;" : "=r"(centred) : "r"(packed), "r"(0x647F647Fu));
                    own.pairs[p] = centred;
                }
                if (lane == 0) own.listed = 0;
                __syncwarp();
                // Visits the estimates of every window of tiles [0, tiles) of the chunk: four per lane and tile of
                // dimensions, windows (row, row + 8) by dimensions (column, column + 1).
                auto sweep = [&](std::uint32_t tiles, auto &&visit) {
                    std::uint32_t at = row + column;
                    std::uint32_t a0 = own.pairs[at], a1, a2;
                    [[maybe_unused]] std::uint32_t a3, a4; // the second 16 bytes
                    if constexpr (steps_ == 2) a1 = own.pairs[at + 8], a2 = own.pairs[at + 16];
                    for (std::uint32_t tile = 0; tile < tiles; ++tile, at += 16) {
                        if constexpr (steps_ == 1) a1 = own.pairs[at + 8], a2 = own.pairs[at + 16];
                        else a3 = own.pairs[at + 24], a4 = own.pairs[at + 32];
                        // A tile's products are issued one tile of dimensions ahead of their epilogue.
                        float hi[2][4], lo[2][4];
                        auto multiply = [&](int t) {
                            mma_tile(hi[t & 1], a0, a1, a1, a2, weights[t][0][0][0], weights[t][0][0][1], bias, bias,
                                     bias, bias);
                            mma_tile(lo[t & 1], a0, a1, a1, a2, weights[t][1][0][0], weights[t][1][0][1], bias, bias,
                                     bias, bias);
                            if constexpr (steps_ == 2) {
                                float(&h)[4] = hi[t & 1], (&l)[4] = lo[t & 1];
                                mma_tile(h, a2, a3, a3, a4, weights[t][0][1][0], weights[t][0][1][1], h[0], h[1], h[2],
                                         h[3]);
                                mma_tile(l, a2, a3, a3, a4, weights[t][1][1][0], weights[t][1][1][1], l[0], l[1], l[2],
                                         l[3]);
                            }
                        };
                        multiply(0);
#pragma unroll
                        for (int t = 0; t < tensor_tiles_k; ++t) {
                            if (t + 1 < tensor_tiles_k) multiply(t + 1);
                            std::uint32_t estimate[4];
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                estimate[j] = __float_as_uint(hi[t & 1][j]) * (1u << 21) +
                                              (__float_as_uint(lo[t & 1][j]) * (1u << 10) + offset[t][j & 1]);
                            visit(tile, t, estimate);
                        }
                        if constexpr (steps_ == 1) a0 = a2;
                        else a0 = a2, a1 = a3, a2 = a4;
                    }
                };
                if (base == 0) {
                    // The first whole tiles bound the minimum: the least estimate, biased down by the margin so that
                    // an estimate wrapped past 2^32 never counts, over the 8 lanes that share a dimension.
                    std::uint32_t least[tensor_tiles_k][2];
#pragma unroll
                    for (int t = 0; t < tensor_tiles_k; ++t) least[t][0] = least[t][1] = 0xFFFFFFFFu;
#pragma unroll
                    for (int t = 0; t < tensor_tiles_k; ++t)
#pragma unroll
                        for (int j = 0; j < 2; ++j) offset[t][j] -= 2 * own.margin[8 * t + column + j];
                    std::uint32_t const whole = (std::uint32_t)min((std::uint64_t)tensor_chunk_k, length - widest + 1);
                    sweep(whole / 16, [&](std::uint32_t, int t, std::uint32_t const (&estimate)[4]) {
                        least[t][0] = min(least[t][0], min(estimate[0], estimate[2]));
                        least[t][1] = min(least[t][1], min(estimate[1], estimate[3]));
                    });
#pragma unroll
                    for (int t = 0; t < tensor_tiles_k; ++t)
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            std::uint32_t const margin = own.margin[8 * t + column + j];
                            offset[t][j] += 2 * margin;
                            std::uint32_t value = least[t][j];
#pragma unroll
                            for (int distance = 4; distance < 32; distance <<= 1)
                                value = min(value, __shfl_xor_sync(0xFFFFFFFFu, value, distance));
                            std::uint32_t const bound = value + 4 * margin;
                            limit[t][j] = bound >= value ? bound : 0xFFFFFFFFu;
                        }
                }
                sweep((here + 15) / 16, [&](std::uint32_t tile, int t, std::uint32_t const (&estimate)[4]) {
                    if (estimate[0] <= limit[t][0] || estimate[1] <= limit[t][1] || estimate[2] <= limit[t][0] ||
                        estimate[3] <= limit[t][1]) {
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            if (estimate[j] > limit[t][j & 1]) continue;
                            std::uint32_t const slot = atomicAdd(&own.listed, 1u);
                            if (slot < tensor_list_k)
                                own.list[slot] = (std::uint16_t)((8 * t + column + (j & 1)) << 8 |
                                                                 (16 * tile + row + 8 * (j >> 1)));
                        }
                    }
                });
                __syncwarp();
            }
            if (own.listed > tensor_list_k) {
                // Exact rolling hashes of the whole chunk, two dimensions per lane side by side.
                __syncwarp();
                rolling_t rolling[2];
                std::uint64_t last[2];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    std::uint32_t const k = lane + 32u * j;
                    bool const any = first_dim + k < dimensions && base + own.width[k] <= length;
                    last[j] = any ? min(base + tensor_chunk_k, length - own.width[k] + 1) : base;
                    rolling[j].open(params[min(first_dim + k, dimensions - 1)], own.minimum[k], own.occurrences[k]);
                    if (any) rolling[j].first(bytes + base);
                }
                std::uint64_t const common = min(last[0], last[1]);
                std::uint8_t const *ahead[2] = {bytes - 1 + rolling[0].width, bytes - 1 + rolling[1].width};
                std::uint64_t p = base + 1;
                for (; p < common; ++p) {
                    std::uint32_t const out = bytes[p - 1];
                    rolling[0].next(out, ahead[0][p]), rolling[1].next(out, ahead[1][p]);
                }
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    for (std::uint64_t rest = p; rest < last[j]; ++rest)
                        rolling[j].next(bytes[rest - 1], ahead[j][rest]);
                    if (last[j] > base)
                        own.minimum[lane + 32 * j] = rolling[j].minimum, own.occurrences[lane + 32 * j] = rolling[j].occurrences;
                }
            }
            else if (own.listed) {
                std::uint32_t const listed = own.listed;
                for (std::uint32_t first = 0; first < listed; first += 32) {
                    std::uint32_t const entry = first + lane < listed ? own.list[first + lane] : 0u;
                    std::uint32_t const dim = entry >> 8, width = own.width[dim];
                    std::uint64_t const window = base + (entry & 255u);
                    unsigned long long const before = own.minimum[dim];
                    unsigned long long value = ~0ull; // no hash: past the list, or past the dimension's last window
                    if (first + lane < listed && window + width <= length) {
                        fingerprint_dim_t const &p = params[min(first_dim + dim, dimensions - 1)];
                        value = window_hash(bytes + window, width, p.multiplier, p.modulo, p.mu);
                    }
                    __syncwarp();
                    if (value < before) atomicMin(&own.minimum[dim], value);
                    __syncwarp();
                    unsigned long long const after = own.minimum[dim];
                    if (after != before) own.occurrences[dim] = 0; // a lower minimum starts its count
                    __syncwarp();
                    if (value == after && value != ~0ull) atomicAdd(&own.occurrences[dim], 1u);
                    __syncwarp();
                }
            }
            else continue;
            // The exact minima's own bounds: minimum * 2^(32 + shift) / m from at most 5 units below, plus twice the
            // margin.
            __syncwarp();
            for (int k = lane; k < tensor_dims_k; k += 32) {
                unsigned long long const minimum = own.minimum[k];
                if (minimum == ~0ull) continue;
                std::uint32_t const fraction =
                    __umulhi((std::uint32_t)((minimum << own.shift[k]) >> 11), own.mu[k]) << 1;
                std::uint32_t const bound = fraction + 8u + 2 * own.margin[k];
                own.limit[k] = bound >= fraction ? bound : 0xFFFFFFFFu;
            }
            __syncwarp();
#pragma unroll
            for (int tile = 0; tile < tensor_tiles_k; ++tile) {
                uint2 const two = *reinterpret_cast<uint2 const *>(&own.limit[8 * tile + column]);
                limit[tile][0] = min(limit[tile][0], two.x), limit[tile][1] = min(limit[tile][1], two.y);
            }
        }
        __syncwarp();
        for (int k = lane; k < tensor_dims_k; k += 32) {
            std::uint32_t const dim = first_dim + k;
            if (dim >= dimensions) continue;
            reinterpret_cast<std::uint32_t *>(reinterpret_cast<unsigned char *>(hashes) + text * hashes_stride)[dim] =
                (std::uint32_t)own.minimum[k]; // no window: all ones
            reinterpret_cast<std::uint32_t *>(reinterpret_cast<unsigned char *>(counts) + text * counts_stride)[dim] =
                own.occurrences[k];
        }
    }
    asm volatile("griddepcontrol.wait;" ::: "memory"); // complete only after the kernels launched before
}

/**
 *  Exact rolling hashes, one warp per text and 32 dimensions: the texts too short for the tensor-core kernel, and every
 *  text of the groups whose windows are too wide for it (a warp passes over the others after a look at their offsets).
 *  Many resident warps hide the serial chain of modular steps, which this path cannot shorten.
 */
__global__ void __launch_bounds__(256, 5) fingerprints_kernel(
    tape_t const texts, fingerprint_dim_t const *__restrict__ params, std::uint32_t const dimensions,
    fingerprint_group_t const *__restrict__ groups, std::uint32_t const groups_count, std::uint32_t const windows_min,
    std::uint32_t *__restrict__ hashes, std::uint64_t const hashes_stride, std::uint32_t *__restrict__ counts,
    std::uint64_t const counts_stride) {
    asm volatile("griddepcontrol.launch_dependents;"); // the tensor-core kernels take other texts: they may start
    int const lane = threadIdx.x & 31;
    std::uint32_t const halves = 2 * groups_count;
    std::uint64_t const items = texts.count * halves;
    std::uint64_t const warps = (std::uint64_t)gridDim.x * (blockDim.x / 32);
    for (std::uint64_t item = (std::uint64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; item < items;
         item += warps) {
        std::uint64_t const text = item / halves;
        std::uint32_t const half = (std::uint32_t)(item % halves);
        fingerprint_group_t const group = groups[half / 2];
        std::uint64_t const start = text_offset(texts, text);
        std::uint64_t const length = text_offset(texts, text + 1) - start;
        if (group.widest <= (std::uint32_t)tensor_width_k && !rolls(length, group.widest, windows_min)) continue;
        std::uint32_t const dim = group.index * fingerprint_group_k + (half & 1u) * 32 + lane;
        bool const live = dim < dimensions;
        if (!__any_sync(0xFFFFFFFFu, live)) continue;
        fingerprint_dim_t const p = params[live ? dim : 0];
        std::uint8_t const *bytes = texts.base + start;
        std::uint32_t min_hash = 0xFFFFFFFFu, min_count = 0;
        if (length >= p.width) {
            // The first window: no outgoing bytes.
            std::uint64_t state = 0;
            for (std::uint32_t i = 0; i < p.width; ++i)
                state = reduce(state * p.multiplier + bytes[i] + 1u, p.modulo, p.mu);
            std::uint64_t minimum = canonical(state, p.modulo);
            std::uint32_t occurrences = 1;
            std::uint32_t const modulo_hi = (std::uint32_t)(p.modulo >> 32);
            std::uint32_t minimum_hi = (std::uint32_t)(minimum >> 32);
            // in + 1 + D * (out + 1) = in + D * out + (D + 1)
            std::uint64_t const constant = p.discard + 1u;
            std::uint64_t const windows = length - p.width;
#pragma unroll 8
            for (std::uint64_t i = 0; i < windows; ++i) {
                std::uint64_t const x =
                    state * p.multiplier + p.discard * bytes[i] + (constant + bytes[p.width + i]);
                state = reduce(x, p.modulo, p.mu);
                std::uint32_t const state_hi = (std::uint32_t)(state >> 32);
                if (__builtin_expect(state_hi <= minimum_hi || state_hi - modulo_hi <= minimum_hi + 1u, 0)) {
                    std::uint64_t const value = canonical(state, p.modulo);
                    if (value <= minimum) {
                        occurrences = value == minimum ? occurrences + 1u : 1u;
                        minimum = value;
                        minimum_hi = (std::uint32_t)(minimum >> 32);
                    }
                }
            }
            min_hash = (std::uint32_t)(minimum & 0xFFFFFFFFu), min_count = occurrences;
        }
        if (live) {
            reinterpret_cast<std::uint32_t *>(reinterpret_cast<unsigned char *>(hashes) + text * hashes_stride)[dim] =
                min_hash;
            reinterpret_cast<std::uint32_t *>(reinterpret_cast<unsigned char *>(counts) + text * counts_stride)[dim] =
                min_count;
        }
    }
}

/** The half-precision bits of an integer of magnitude at most 2,048 (exact). */
std::uint16_t half_bits(int value) {
    if (!value) return 0;
    unsigned const magnitude = (unsigned)std::abs(value);
    int exponent = 0;
    while (magnitude >> (exponent + 1)) ++exponent;
    unsigned const fraction = exponent <= 10 ? (magnitude << (10 - exponent)) & 1023u : 0u; // 2,048 = 2^11
    return (std::uint16_t)((value < 0 ? 0x8000u : 0u) | (unsigned)(exponent + 15) << 10 | fraction);
}

std::uint64_t splitmix64(std::uint64_t state) {
    state += 0x9E3779B97F4A7C15ull;
    std::uint64_t z = state;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

} // namespace

fingerprint_dim_t fingerprint_dimension(std::uint64_t dim, std::uint64_t width, std::uint64_t seed,
                                        fingerprint_weights_t &weights) {
    fingerprint_dim_t p {};
    weights = {};
    // Parameters of the reference's `floating_rolling_hasher<f64_t>` (serial.hpp:426-432).
    p.multiplier = (std::uint32_t)(256u + splitmix64(seed + dim) % 384u);
    p.modulo = 4503599626977ull - splitmix64(splitmix64(seed + dim)) % (1ull << 20);
    std::uint64_t leading = 1; // a^(w-1) mod m: the weight of a window's oldest byte
    for (std::uint64_t i = 0; i + 1 < width; ++i) leading = leading * p.multiplier % p.modulo;
    p.discard = (p.modulo - leading * p.multiplier % p.modulo) % p.modulo;
    p.mu = (std::uint32_t)(((unsigned __int128)1 << 74) / p.modulo);
    p.width = (std::uint32_t)width;
    if (width <= (std::uint64_t)tensor_width_k) {
        // Weights a^(w-1-i) / m in units of 2^-22, rounded, as two signed digits of 11 bits; the margin bounds what the
        // rounding can cost a window of centred bytes (at most 128 in magnitude), in units of 2^-32.
        // Short windows whose hashes never reach the modulus are scaled up to fill it.
        std::uint64_t weight = 1, sum = 0, largest = 0; // largest: 256 * sum of a^k, until it passes m
        for (std::uint64_t k = 0; k < width && largest < p.modulo; ++k) largest = largest * p.multiplier + 256u;
        while (largest << (p.shift + 1) < p.modulo) ++p.shift;
        double error = 0;
        for (std::uint64_t k = 0; k < width; ++k) {
            std::uint64_t const i = width - 1 - k;
            auto const scaled = (unsigned __int128)weight << (22 + p.shift);
            std::uint64_t const rounded = (std::uint64_t)((scaled + p.modulo / 2) / p.modulo);
            auto const difference = (__int128)rounded * p.modulo - (__int128)scaled; // at most m / 2 in magnitude
            error += std::abs((double)difference) / (double)p.modulo * 1024.0;
            int const low = (int)((rounded + 1024) & 2047) - 1024;
            int const high = (int)((((rounded - (std::uint64_t)(std::int64_t)low) >> 11) + 1024) & 2047) - 1024;
            weights.digits[0][i] = half_bits(high), weights.digits[1][i] = half_bits(low);
            sum = (sum + weight) % p.modulo;
            weight = weight * p.multiplier % p.modulo;
        }
        p.margin = (std::uint32_t)std::ceil(128.0 * error) + 8u;
        p.offset = (std::uint32_t)(((unsigned __int128)(sum * 128 % p.modulo) << (32 + p.shift)) / p.modulo);
    }
    return p;
}

fingerprint_groups_t fingerprint_groups(fingerprint_dim_t const *params, std::uint32_t dimensions,
                                        fingerprint_group_t *groups) {
    fingerprint_groups_t made {};
    std::uint32_t const total = (dimensions + tensor_dims_k - 1) / tensor_dims_k;
    std::uint32_t cursor = 0;
    for (int kind = 0; kind < 3; ++kind)
        for (std::uint32_t group = 0; group < total; ++group) {
            std::uint32_t widest = 0;
            for (std::uint32_t d = group * tensor_dims_k; d < std::min(dimensions, (group + 1) * tensor_dims_k); ++d)
                widest = std::max(widest, params[d].width);
            if ((widest <= 16 ? 0 : widest <= (std::uint32_t)tensor_width_k ? 1 : 2) != kind) continue;
            groups[cursor++] = {group, widest}, ++made.count[kind];
        }
    return made;
}

cudaError_t launch_fingerprints(tape_t const &texts, fingerprint_dim_t const *params,
                                fingerprint_weights_t const *weights, std::uint32_t dimensions,
                                fingerprint_group_t const *group_list, fingerprint_groups_t const &groups,
                                std::uint32_t *hashes, std::uint64_t hashes_stride, std::uint32_t *counts,
                                std::uint64_t counts_stride, int sm_count, cudaStream_t stream) {
    if (!texts.count || !dimensions) return cudaSuccess;
    // The kernels divide the texts and groups among themselves, so each may start as soon as the one before has all its
    // CTAs running: their tails overlap, and one without a text of its own costs a look at the offsets.
    std::uint32_t const total = groups.count[0] + groups.count[1] + groups.count[2];
    std::uint64_t const blocks = (texts.count * 2 * total + 7) / 8; // 8 warps per CTA
    unsigned const grid = (unsigned)std::min<std::uint64_t>(blocks, (std::uint64_t)sm_count * 16);
    std::uint32_t const windows_min = tensor_windows_min(texts.count * total, sm_count);
    fingerprints_kernel<<<grid, 256, 0, stream>>>(texts, params, dimensions, group_list, total, windows_min, hashes,
                                                  hashes_stride, counts, counts_stride);
    cudaError_t launched = cudaGetLastError();
    cudaLaunchAttribute overlap;
    overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    overlap.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config = {};
    config.stream = stream;
    config.attrs = &overlap, config.numAttrs = 1;
    // Wider windows first: their warps take longest.
    for (int kind = 1; kind >= 0 && launched == cudaSuccess; --kind) {
        std::uint32_t const here = groups.count[kind];
        if (!here) continue;
        fingerprint_group_t const *list = group_list + (kind ? groups.count[0] : 0);
        // One warp per CTA while that spreads the work over more SMs; at least one warp per group, so that every group
        // has a slot.
        std::uint64_t const items = texts.count * here;
        int const warps = items <= (std::uint64_t)sm_count * tensor_warps_k ? 1 : tensor_warps_k;
        std::uint64_t const resident = (std::uint64_t)sm_count * (kind == 0 ? 4 : 3) * tensor_warps_k;
        std::uint64_t const wanted = std::max<std::uint64_t>(std::min(items, resident / here * here), here);
        config.gridDim = dim3((unsigned)((wanted + warps - 1) / warps));
        config.blockDim = dim3(32 * warps);
        config.dynamicSmemBytes = sizeof(tensor_warp_t) * (std::size_t)warps;
        launched = cudaLaunchKernelEx(
            &config, kind == 0 ? fingerprints_tensor_kernel<1> : fingerprints_tensor_kernel<2>, texts, params, weights,
            dimensions, list, here, windows_min, hashes, hashes_stride, counts, counts_stride);
    }
    return launched;
}

} // namespace szs_gb300
