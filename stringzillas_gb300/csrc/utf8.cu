/**
 *  @file utf8.cu
 *  @brief UTF-8 Levenshtein: code points of both tapes transcoded to one-byte codes on the device.
 *
 *  Edit distances over code points depend only on which code points are equal, so the batch's distinct code points
 *  are numbered 0..k-1 and every string is rewritten as a string of those numbers: bytes when k <= 256 (the byte-level
 *  Levenshtein routes then score the transcoded tapes unchanged), 16-bit codes up to k = 65,536 (scored by the
 *  Levenshtein routes' 16-bit-symbol instances). The reference decodes each string rune by rune
 *  (include/stringzillas/similarities/serial.hpp:2288-2299) with `sz_rune_decode_unchecked`
 *  (include/stringzilla/utf8_runes/serial.h:101-115): the length comes from the lead byte alone and continuation
 *  bytes are not checked, so a sequence cut off by the end of a string reads on into the next string of the tape.
 *  The same rule is applied here; bytes past the end of the tape read as 0.
 *
 *  Passes: (1) one warp per string walks its code points, counts them, marks each in a bitmap (a CTA marks the Basic
 *  Multilingual Plane in shared memory, 8 KB, and merges what the global bitmap lacks at its end; rarer code points are
 *  marked in the global bitmap directly) and writes them as 16-bit values, from the code unit of the string's first byte
 *  on, so no scan of the counts is needed and the tapes keep their offsets beside the counts as lengths. (2) One CTA
 *  ranks the bitmap's words, so a code point's rank is the number of distinct code points below it. A call over more
 *  than 256 code points, all inside that plane, is then done: its codes are the code points. (3) Calls over at most 256
 *  are recoded from the 16-bit values to one-byte ranks, and calls with code points beyond the plane walk their strings
 *  again and write ranks. 65,536 pairs of 100-300 CJK ideographs (79.7 MB): 0.72 ms with a counting and a writing walk,
 *  a scan and byte loads, 0.20 ms now.
 */
#include "launchers.h"

namespace szs_gb300 {

namespace {

__device__ __forceinline__ std::uint32_t rune_at(std::uint8_t const *base, std::uint64_t position, std::uint64_t end,
                                                 std::uint32_t &length) {
    std::uint32_t const lead = base[position];
    length = 1u + (lead >= 0xC0u) + (lead >= 0xE0u) + (lead >= 0xF0u);
    auto next = [&](std::uint32_t k) -> std::uint32_t {
        return position + k < end ? (std::uint32_t)(base[position + k] & 0x3Fu) : 0u;
    };
    switch (length) {
    case 1: return lead;
    case 2: return (lead & 0x1Fu) << 6 | next(1);
    case 3: return (lead & 0x0Fu) << 12 | next(1) << 6 | next(2);
    default: return (lead & 0x07u) << 18 | next(1) << 12 | next(2) << 6 | next(3);
    }
}

__device__ __forceinline__ std::uint64_t tape_offset(tape_t const &tape, std::uint64_t i) {
    return tape.offset_bits == 32 ? static_cast<std::uint32_t const *>(tape.offsets)[i]
                                  : static_cast<std::uint64_t const *>(tape.offsets)[i];
}

constexpr std::uint32_t plane_words_k = 65536 / 32; // the Basic Multilingual Plane's 2,048 bitmap words
constexpr int utf8_threads_k = 128;

/**
 *  One warp walks the string [begin, stop) 128 bytes at a time, lane L on bytes 4L..4L+3 of each window (from aligned
 *  words, shifted to the string's own alignment), and calls `visit(rune, index)` once per code point, `index` counting
 *  code points from the string's start: consecutive lanes hold consecutive code points. This holds only when the string
 *  is well formed in the decoder's sense: its continuation bytes (10xxxxxx) are exactly those that its lead bytes ask
 *  for, the byte after every lead of 0xC0 or more, the second after 0xE0 or more and the third after 0xF0 or more, none
 *  past `stop`; then the code points start exactly at the other bytes, as a sequential walk would find them. Returns
 *  false, warp-uniformly, as soon as a window breaks that, or for strings of 2^31 bytes or more; both passes then walk the
 *  whole string again sequentially. Code points visited before stay visited, so each has to be one that this walk finds
 *  too: windows before a broken one are, and a sequence that leaves its window is decoded there only if the string holds
 *  all of its bytes (the sequential walk reads on into the next string). Sets `count` to the string's code points on
 *  success. `positions`: 128 bytes of shared memory of the warp's own.
 */
template <typename visit_>
__device__ __forceinline__ bool warp_walk(tape_t const &tape, std::uint64_t begin, std::uint64_t stop,
                                          std::uint8_t *positions, std::uint64_t &count, visit_ &&visit) {
    if (stop - begin >= (1ull << 31)) return false;
    std::uint32_t const n = (std::uint32_t)(stop - begin);
    count = 0;
    if (!n) return true;
    std::uintptr_t const address = reinterpret_cast<std::uintptr_t>(tape.base + begin);
    std::uint32_t const *aligned = reinterpret_cast<std::uint32_t const *>(address & ~std::uintptr_t(3));
    std::uint32_t const skew = (std::uint32_t)(address & 3), last = (skew + n - 1) >> 2;
    int const lane = threadIdx.x & 31;
    std::uint32_t const lower = (1u << lane) - 1u;
    std::uint32_t runes = 0;
    std::uint32_t asked = 0; // lane 0: continuation bytes that the last window's leads ask of this window's first bytes
    for (std::uint32_t window = 0; window < n; window += 128) {
        std::uint32_t const at = window / 4 + lane;
        std::uint32_t const a = __ldg(aligned + min(at, last)), b = __ldg(aligned + min(at + 1, last)),
                            c = __ldg(aligned + min(at + 2, last));
        std::uint32_t own = __funnelshift_r(a, b, 8 * skew);
        std::uint32_t const high = __funnelshift_r(b, c, 8 * skew); // read only where a sequence goes on
        std::uint32_t valid = 0x80808080u;
        std::uint32_t outside = 0; // lane 31: which of the three bytes after this window lie past the string
        if (window + 130 >= n) {
            std::uint32_t const left = n - min(window + 128, n); // at most 2
            outside = lane == 31 ? 0x00FFFFFFu << (8 * left) : 0u;
            int const keep = (int)n - (int)(window + 4 * lane); // this lane's bytes inside the string
            std::uint32_t const mask = keep >= 4 ? 0xFFFFFFFFu : (keep <= 0 ? 0u : 0xFFFFFFFFu >> (32 - 8 * keep));
            own &= mask, valid &= mask;
        }
        if (!__any_sync(0xFFFFFFFFu, (own & 0x80808080u) | asked)) { // ASCII
            std::uint32_t const total = min(128u, n - window);
#pragma unroll
            for (std::uint32_t k = 0; k < 128; k += 32) {
                std::uint32_t const p = k + lane;
                std::uint32_t const word = __shfl_sync(0xFFFFFFFFu, own, p >> 2);
                if (p < total) visit(__byte_perm(word, 0u, 0x4440u + (p & 3u)), (std::uint64_t)(runes + p));
            }
            runes += total;
            continue;
        }
        // Per byte, in its top bit: continuation bytes, and leads of two, three and four bytes.
        std::uint32_t const continuation = own & ~(own << 1) & 0x80808080u;
        std::uint32_t const two = own & (own << 1) & 0x80808080u, three = two & (own << 2), four = three & (own << 3);
        std::uint32_t const here = two << 8 | three << 16 | four << 24, beyond = two >> 24 | three >> 16 | four >> 8;
        std::uint32_t const above = __shfl_up_sync(0xFFFFFFFFu, beyond, 1);
        bool const broken = (here | (lane ? above : asked)) != continuation || (beyond & outside);
        std::uint32_t const carried = __shfl_sync(0xFFFFFFFFu, beyond, 31);
        asked = lane ? 0u : carried;
        if (__any_sync(0xFFFFFFFFu, broken)) return false;
        std::uint32_t const leads = (((valid & ~continuation) >> 7) * 0x01020408u) >> 24; // four bits
        // The window's code points in order: their positions, so that lane k takes the k-th.
        std::uint32_t const found = __popc(leads);
        std::uint32_t const ones = __ballot_sync(0xFFFFFFFFu, found & 1u), twos = __ballot_sync(0xFFFFFFFFu, found & 2u),
                            fours = __ballot_sync(0xFFFFFFFFu, found & 4u);
        std::uint32_t const before = __popc(ones & lower) + 2u * __popc(twos & lower) + 4u * __popc(fours & lower);
        std::uint32_t const total = __popc(ones) + 2u * __popc(twos) + 4u * __popc(fours);
#pragma unroll
        for (std::uint32_t j = 0; j < 4; ++j)
            if ((leads >> j) & 1u) positions[before + __popc(leads & ((1u << j) - 1u))] = (std::uint8_t)(4 * lane + j);
        __syncwarp();
        for (std::uint32_t k = 0; k < total; k += 32) {
            bool const live = k + lane < total;
            std::uint32_t const p = live ? positions[k + lane] : 0u;
            std::uint32_t const low_word = __shfl_sync(0xFFFFFFFFu, own, p >> 2);
            std::uint32_t const high_word = __shfl_sync(0xFFFFFFFFu, high, p >> 2);
            // The lead byte on top, then the three bytes after it; a sequence's bits are the top ones of 6 + 18.
            std::uint32_t const bytes = __byte_perm(low_word, high_word, 0x0123u + 0x1111u * (p & 3u));
            std::uint32_t const lead = bytes >> 24;
            std::uint32_t const more = (lead >= 0xC0u) + (lead >= 0xE0u) + (lead >= 0xF0u);
            std::uint32_t const sixes = bytes & 0x3F3F3F3Fu;
            std::uint32_t const twelves = ((sixes >> 2) & 0x0FC00FC0u) | (sixes & 0x003F003Fu);
            std::uint32_t const all = (twelves >> 16) << 12 | (twelves & 0xFFFu);
            std::uint32_t const rune = more ? (all >> (18 - 6 * more)) & ((1u << (5 * more + 6)) - 1u) : lead;
            if (live) visit(rune, (std::uint64_t)(runes + k + lane));
        }
        __syncwarp();
        runes += total;
    }
    count = runes;
    return true;
}

/** Pass 1: code points per string, the bitmap, and the code points as 16-bit values (truncated beyond the Basic
 *  Multilingual Plane, which sets `set->beyond`): one warp per string, written at `out` + its offset from the tape's
 *  first. */
__global__ void __launch_bounds__(utf8_threads_k) utf8_decode_kernel(tape_t const tape, std::uint64_t const end,
                                                                     std::uint64_t *__restrict__ counts,
                                                                     rune_set_t *__restrict__ set,
                                                                     std::uint16_t *__restrict__ out) {
    __shared__ std::uint32_t plane_s[plane_words_k];
    __shared__ std::uint8_t positions_s[utf8_threads_k / 32][128];
    for (std::uint32_t k = threadIdx.x; k < plane_words_k; k += blockDim.x) plane_s[k] = 0u;
    __syncthreads();
    auto mark = [&](std::uint32_t rune) {
        std::uint32_t const bit = 1u << (rune & 31u);
        if (rune < 65536u) {
            if (!(plane_s[rune >> 5] & bit)) atomicOr(&plane_s[rune >> 5], bit);
        }
        else {
            atomicOr(&set->present[rune >> 5], bit);
            set->beyond = 1u;
        }
    };
    int const lane = threadIdx.x & 31;
    std::uint64_t const first = tape_offset(tape, 0);
    std::uint64_t const warps = (std::uint64_t)gridDim.x * (blockDim.x >> 5);
    for (std::uint64_t i = (std::uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < tape.count;
         i += warps) {
        std::uint64_t const begin = tape_offset(tape, i), stop = tape_offset(tape, i + 1);
        std::uint16_t *target = out + (begin - first);
        std::uint64_t runes = 0;
        bool const walked = warp_walk(tape, begin, stop, positions_s[threadIdx.x >> 5], runes,
                                      [&](std::uint32_t rune, std::uint64_t index) {
                                          mark(rune);
                                          target[index] = (std::uint16_t)rune;
                                      });
        __syncwarp();
        if (!walked && lane == 0) { // the decoder's sequential rule, as the reference applies it
            runes = 0;
            for (std::uint64_t position = begin; position < stop; ++runes) {
                std::uint32_t length;
                std::uint32_t const rune = rune_at(tape.base, position, end, length);
                mark(rune);
                target[runes] = (std::uint16_t)rune;
                position += length;
            }
        }
        if (lane == 0) counts[i] = runes;
    }
    __syncthreads();
    for (std::uint32_t k = threadIdx.x; k < plane_words_k; k += blockDim.x)
        if (plane_s[k] & ~__ldcg(&set->present[k])) atomicOr(&set->present[k], plane_s[k]);
}

/** Pass 2: the rank of every bitmap word and the number of distinct code points (one CTA of 32 warps, each over a
 *  contiguous block of words read 32 at a time): the Basic Multilingual Plane's words, and all 65,536 only when a code
 *  point beyond it was marked. */
__global__ void __launch_bounds__(1024) utf8_codes_kernel(rune_set_t *__restrict__ set) {
    constexpr int warps = 32;
    std::uint32_t const per_warp = (set->beyond ? rune_words_k : plane_words_k) / warps;
    __shared__ std::uint32_t warp_totals[warps];
    int const lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    std::uint32_t const *present = set->present + warp * per_warp;
    std::uint32_t *rank = set->rank + warp * per_warp;
    std::uint32_t sum = 0;
    for (std::uint32_t k = lane; k < per_warp; k += 32) sum += __popc(present[k]);
    sum = __reduce_add_sync(0xFFFFFFFFu, sum);
    if (lane == 0) warp_totals[warp] = sum;
    __syncthreads();
    std::uint32_t offset = 0; // distinct code points in the blocks before this warp's
    for (int w = 0; w < warp; ++w) offset += warp_totals[w];
    for (std::uint32_t base = 0; base < per_warp; base += 32) {
        std::uint32_t const own = __popc(present[base + lane]);
        std::uint32_t scan = own; // inclusive over the 32 words
#pragma unroll
        for (int distance = 1; distance < 32; distance <<= 1) {
            std::uint32_t const lower = __shfl_up_sync(0xFFFFFFFFu, scan, distance);
            if (lane >= distance) scan += lower;
        }
        rank[base + lane] = offset + scan - own;
        offset += __shfl_sync(0xFFFFFFFFu, scan, 31);
    }
    if (threadIdx.x == 0) {
        std::uint32_t symbols = 0;
        for (int w = 0; w < warps; ++w) symbols += warp_totals[w];
        set->symbols = symbols;
    }
}

/** A string's room past its codes, filled with code 0 (one of the batch's, so that an alphabet pass over the tape's whole
 *  range sees no other symbols). */
__device__ __forceinline__ void fill_room(std::uint8_t *target, std::uint64_t codes, std::uint64_t room, int lane) {
    for (std::uint64_t k = codes + lane; k < room; k += 32) target[k] = 0;
}

/** Pass 3, at most 256 code points, none beyond the plane: each string's 16-bit values as one-byte ranks. */
__global__ void __launch_bounds__(utf8_threads_k)
    utf8_recode_kernel(tape_t const tape, std::uint64_t const *__restrict__ counts, rune_set_t const *__restrict__ set,
                       std::uint16_t const *__restrict__ values, std::uint8_t *__restrict__ out) {
    __shared__ std::uint32_t present_s[plane_words_k], rank_s[plane_words_k];
    for (std::uint32_t k = threadIdx.x; k < plane_words_k; k += blockDim.x)
        present_s[k] = set->present[k], rank_s[k] = set->rank[k];
    __syncthreads();
    int const lane = threadIdx.x & 31;
    std::uint64_t const first = tape_offset(tape, 0);
    std::uint64_t const warps = (std::uint64_t)gridDim.x * (blockDim.x >> 5);
    for (std::uint64_t i = (std::uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < tape.count;
         i += warps) {
        std::uint64_t const begin = tape_offset(tape, i), room = tape_offset(tape, i + 1) - begin, codes = counts[i];
        std::uint16_t const *source = values + (begin - first);
        std::uint8_t *target = out + (begin - first);
        for (std::uint64_t k = lane; k < codes; k += 32) {
            std::uint32_t const rune = source[k];
            target[k] = (std::uint8_t)(rank_s[rune >> 5] + __popc(present_s[rune >> 5] & ((1u << (rune & 31u)) - 1u)));
        }
        fill_room(target, codes, room, lane);
    }
}

/** Pass 3, calls with code points beyond the plane: each string's ranks (one byte each, or two for more than 256 code
 *  points), one warp per string. */
template <typename code_type_>
__global__ void __launch_bounds__(utf8_threads_k)
    utf8_write_kernel(tape_t const tape, std::uint64_t const end, std::uint64_t const *__restrict__ counts,
                      rune_set_t const *__restrict__ set, code_type_ *__restrict__ out) {
    __shared__ std::uint32_t present_s[plane_words_k], rank_s[plane_words_k];
    __shared__ std::uint8_t positions_s[utf8_threads_k / 32][128];
    for (std::uint32_t k = threadIdx.x; k < plane_words_k; k += blockDim.x)
        present_s[k] = set->present[k], rank_s[k] = set->rank[k];
    __syncthreads();
    auto code_of = [&](std::uint32_t rune) -> std::uint32_t {
        std::uint32_t const word = rune >> 5, below = (1u << (rune & 31u)) - 1u;
        return rune < 65536u ? rank_s[word] + __popc(present_s[word] & below)
                             : __ldg(set->rank + word) + __popc(__ldg(set->present + word) & below);
    };
    int const lane = threadIdx.x & 31;
    std::uint64_t const first = tape_offset(tape, 0);
    std::uint64_t const warps = (std::uint64_t)gridDim.x * (blockDim.x >> 5);
    for (std::uint64_t i = (std::uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < tape.count;
         i += warps) {
        std::uint64_t const begin = tape_offset(tape, i), stop = tape_offset(tape, i + 1);
        code_type_ *const target = out + (begin - first);
        std::uint64_t runes = 0;
        bool const walked = warp_walk(tape, begin, stop, positions_s[threadIdx.x >> 5], runes,
                                      [&](std::uint32_t rune, std::uint64_t index) {
                                          target[index] = (code_type_)code_of(rune);
                                      });
        __syncwarp();
        if (!walked && lane == 0) { // the decoder's sequential rule, as the reference applies it
            code_type_ *next = target;
            for (std::uint64_t position = begin; position < stop;) {
                std::uint32_t length;
                *next++ = (code_type_)code_of(rune_at(tape.base, position, end, length));
                position += length;
            }
        }
        if constexpr (sizeof(code_type_) == 1) fill_room(target, counts[i], stop - begin, lane);
    }
}

/** Both tapes' first and last offsets, into page-locked host memory. */
__global__ void utf8_extents_kernel(tape_t const queries, tape_t const candidates, std::uint64_t *__restrict__ extents) {
    tape_t const &tape = threadIdx.x < 2 ? queries : candidates;
    if (threadIdx.x < 4) extents[threadIdx.x] = tape_offset(tape, threadIdx.x & 1 ? tape.count : 0);
}

} // namespace

static int utf8_grid(std::uint64_t strings, int sm_count) {
    std::uint64_t const blocks = (strings + utf8_threads_k / 32 - 1) / (utf8_threads_k / 32); // a warp per string
    return (int)(blocks < (std::uint64_t)sm_count * 16 ? blocks : (std::uint64_t)sm_count * 16);
}

cudaError_t launch_utf8_extents(tape_t const &queries, tape_t const &candidates, std::uint64_t *extents,
                                cudaStream_t stream) {
    utf8_extents_kernel<<<1, 32, 0, stream>>>(queries, candidates, extents);
    return cudaGetLastError();
}

cudaError_t launch_utf8_decode(tape_t const &tape, std::uint64_t end, std::uint64_t *counts, rune_set_t *set,
                               std::uint16_t *values, int sm_count, cudaStream_t stream) {
    if (!tape.count) return cudaSuccess;
    utf8_decode_kernel<<<utf8_grid(tape.count, sm_count), utf8_threads_k, 0, stream>>>(tape, end, counts, set, values);
    return cudaGetLastError();
}

cudaError_t launch_utf8_codes(rune_set_t *set, cudaStream_t stream) {
    utf8_codes_kernel<<<1, 1024, 0, stream>>>(set);
    return cudaGetLastError();
}

cudaError_t launch_utf8_recode(tape_t const &tape, std::uint64_t const *counts, rune_set_t const *set,
                               std::uint16_t const *values, std::uint8_t *out, int sm_count, cudaStream_t stream) {
    if (!tape.count) return cudaSuccess;
    utf8_recode_kernel<<<utf8_grid(tape.count, sm_count), utf8_threads_k, 0, stream>>>(tape, counts, set, values, out);
    return cudaGetLastError();
}

cudaError_t launch_utf8_write(tape_t const &tape, std::uint64_t end, std::uint64_t const *counts, rune_set_t const *set,
                              void *out, bool wide, int sm_count, cudaStream_t stream) {
    if (!tape.count) return cudaSuccess;
    int const grid = utf8_grid(tape.count, sm_count);
    if (wide)
        utf8_write_kernel<<<grid, utf8_threads_k, 0, stream>>>(tape, end, counts, set, static_cast<std::uint16_t *>(out));
    else
        utf8_write_kernel<<<grid, utf8_threads_k, 0, stream>>>(tape, end, counts, set, static_cast<std::uint8_t *>(out));
    return cudaGetLastError();
}

} // namespace szs_gb300
