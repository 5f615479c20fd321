/**
 *  @file direct_rule.h
 *  @brief Which unit-cost cross products the direct kernels (direct.cu) score, and with which side as the patterns.
 *
 *  A direct kernel's warp scores one pattern against 32 consecutive texts and lasts as long as the longest of them, and a
 *  CTA prepares a table per pattern, so what it costs depends on the lengths in input order and on the counts. The planned
 *  routes bin pairs by length and spread them over warps one by one, but plan, and take the slower warp-per-pair kernel for
 *  shorter sides past 512. Both are estimated in word-columns (one 32-row word over one text symbol, ten operations):
 *
 *      direct    0.88 x sum of the patterns' words (in the steps of their class) x sum of the texts' lengths, each padded
 *                to the longest of its 32, + per cell + per table;
 *      planned   sum of words of the shorter side x sum of lengths of the longer one, three times as much again for the
 *                cells whose sides both pass 512, + per pair + per call;
 *      either    at least one thread's (or warp's) chain over the longest text: 25 ns a column at one word and 325 at 32
 *                direct, 21 at one and 190 to 250 at 16 planned, 90 in the warp-per-pair kernel.
 *
 *  Fitted to whole calls on a GB300, which does about 1.56e12 word-columns a second planned and an eighth more direct
 *  (800,000 pairs of 150 x 150: 457 us direct with six words each, 495 planned with five). With the queries as patterns
 *  whenever they fit, 1,000,000 x 1 strings of 150 took 25.4 ms against 0.60 planned (0.57 by this rule), 1,024 x 1,024 of
 *  which 3 % have 1,000 symbols and the others 20 2.86 ms against 0.53, and 2,048 x 2,048 of log-normal lengths (median 100,
 *  sigma 0.7) 7.0 ms against 2.2.
 */
#pragma once
#include <algorithm>
#include <cstdint>

namespace szs_gb300 {

constexpr std::uint64_t direct_max_rows_k = 1024; // longest pattern of the direct cross-product kernels
/** Fewest cells of a cross product for the direct kernels with patterns of 513 to 1,024 rows: one thread per cell takes
 *  about 0.33 ms for a pair of 1,000 bytes however few there are, where the warp-per-pair kernel spreads few pairs over
 *  more SMs (256 pairs 0.28 ms, 2,560 0.45 ms, 3,600 0.54 ms). */
constexpr std::uint64_t direct_min_pairs_k = 1536;

/** Word-columns that the whole GPU scores in a nanosecond on the planned routes. */
constexpr double direct_columns_per_ns_k = 1560;

/** What the rule reads of a tape's lengths; each part of a tape has its own and they add up (`longest`: the largest). */
struct direct_extents_t {
    std::uint64_t longest;     // at most 2^32 - 1
    std::uint64_t symbols;     // sum of the lengths
    std::uint64_t padded;      // the same with every string as long as the longest of its 32 (input order, from a multiple)
    std::uint64_t words;       // 32-row words
    std::uint64_t words_two;   // words in steps of two and of four, as the kernels of longer patterns take them
    std::uint64_t words_four;
    std::uint64_t long_words;  // words of the strings past 512
};

enum direct_choice_t : int {
    direct_none_k = 0,       // the planned routes
    direct_queries_k = 1,    // patterns: the queries
    direct_candidates_k = 2, // patterns: the candidates
};

/** Word-columns of a direct kernel with these patterns and texts, or a negative number where there is none. */
inline double direct_cost(direct_extents_t const &patterns, std::uint64_t patterns_count, direct_extents_t const &texts,
                          std::uint64_t texts_count) {
    if (patterns.longest > direct_max_rows_k || texts.longest >= (1ull << 31)) return -1;
    if (patterns.longest > 512 && (double)patterns_count * (double)texts_count < (double)direct_min_pairs_k) return -1;
    double const words = (double)(patterns.longest <= 128   ? patterns.words
                                  : patterns.longest <= 512 ? patterns.words_two
                                                            : patterns.words_four);
    double const cells = (double)patterns_count * (double)((texts_count + 31) / 32 * 32);
    double const tables = (double)patterns_count * (double)((texts_count + 1023) / 1024);
    double const chain = (double)texts.longest * (15 + 9.7 * (double)((patterns.longest + 31) / 32));
    return std::max(0.88 * words * (double)texts.padded + 22 * cells + 8000 * tables, direct_columns_per_ns_k * chain);
}

/** The same of the planned routes. */
inline double planned_cost(direct_extents_t const &queries, std::uint64_t queries_count,
                           direct_extents_t const &candidates, std::uint64_t candidates_count) {
    bool const shorter_queries =
        (double)queries.symbols * (double)candidates_count <= (double)candidates.symbols * (double)queries_count;
    double const cells = (shorter_queries ? (double)queries.words * (double)candidates.symbols
                                          : (double)candidates.words * (double)queries.symbols) +
                         3 * 32 * (double)queries.long_words * (double)candidates.long_words;
    std::uint64_t const rows = std::min(queries.longest, candidates.longest);
    double const chain = (double)std::max(queries.longest, candidates.longest) *
                         (rows <= 512 ? 9 + 11.4 * (double)((rows + 31) / 32) : 90);
    return std::max(cells, direct_columns_per_ns_k * chain) + 86 * (double)queries_count * (double)candidates_count + 9.4e7;
}

inline direct_choice_t direct_choice(direct_extents_t const &queries, std::uint64_t queries_count,
                                     direct_extents_t const &candidates, std::uint64_t candidates_count) {
    double const by_queries = direct_cost(queries, queries_count, candidates, candidates_count);
    double const by_candidates = direct_cost(candidates, candidates_count, queries, queries_count);
    // Candidates as patterns write down the matrix's columns: only where they save something.
    bool const swapped = by_candidates >= 0 && (by_queries < 0 || by_candidates < 0.97 * by_queries);
    double const best = swapped ? by_candidates : by_queries;
    if (best < 0 || best > planned_cost(queries, queries_count, candidates, candidates_count)) return direct_none_k;
    return swapped ? direct_candidates_k : direct_queries_k;
}

} // namespace szs_gb300
