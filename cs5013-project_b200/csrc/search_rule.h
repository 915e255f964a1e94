// search_rule.h -- which search kernel a batch gets: a CTA or a warp per query, and the
// launch-bound variant of the warp kernels.  Plain C++, no device types.
#pragma once
#include <cstdint>

namespace vann {

struct SearchShape {
    uint64_t nq;
    uint32_t D, R, L, beam;
    int      store;        // vann_store: 0 FP32, 1 BF16, 2 FP8, 3 uint8, 4 PQ
    bool     int_queries;  // build and insert searches over the exact uint8 copy
};

// Batches served by a CTA per query (search_cta.cuh): up to as many queries as keep it
// ahead of a warp per query, which needs many to fill the chip but then does more of them.
// Measured on 148 SMs, CTA / warp per query in us:
//   worklist in registers otherwise (L <= 64): uint8 1M x 128, L = 64: 1 query 88 / 114, 300
//     queries 247 / 305, 590 322 / 373; uint8 L = 32: 1 query 50 / 58, 590 114 / 134 (with 8
//     rows a round instead of 4, 700 queries took 148 / 135);
//   L <= 128, or wider rows or lists: FP32 200k x 96, L = 100: 1 query 116 / 211, 590 298 /
//     479, 1,000 365 / 481 (1,200: 494 / 476); BF16 100k x 256, L = 128 with rerank: 1 query
//     242 / 493, 590 563 / 981, 1,000 837 / 1,074 (1,200: 1,126 / 1,110).  The warp kernel's
//     time over the CTA's with rows of 384 and 512 dimensions and with R = 96 and 128, every
//     format, L = 32 to 100: 1.6 to 4.2 up to 590 queries, 0.97 (uint8 x 96, R = 96, L = 100)
//     to 2.6 at 1,036;
//   L <= 256 (more registers, fewer CTAs): FP32 L = 200: 1 query 189 / 319, 300 239 / 416 (590:
//     451 / 429); the wider shapes above at L = 200: 1.6 to 3.6 times up to 440 queries.
inline bool cta_per_query(const SearchShape& s, int sms) {
    if (s.store == 4 || s.beam == 2 || s.L > 256) return false;
    const uint64_t per_sm = s.L > 128 ? 3 : (s.L > 64 || s.D > 128 || s.R > 64 ? 7 : 4);
    return s.nq <= per_sm * (uint64_t)sms;
}

// Launch-bound variants (blocks of 4 warps per SM) by their index.
constexpr int kBlocks6 = 0, kBlocks4 = 1, kBlocks5 = 2, kBlocks7 = 3, kBlocks8 = 4;

// Launch-bound variant of a warp-per-query search that was not autotuned.  A register cap
// trades resident warps for spills and L1 for filters, so the choice depends on the row
// format's registers, on the list length (shared memory) and on how many warps the batch can
// fill: while every query is resident, more registers cost nothing.  Times relative to 6
// blocks, over indexes of 10k to 1M rows, D = 64 to 128, R = 32 to 64, L = 32 to 500 (mean, and
// the worst index where it is above 1):
//   every query resident at 4 blocks (16 per SM): 4.  uint8 0.95, FP32 0.98, BF16 0.97;
//   FP8 otherwise (its conversions need the registers): 5, R = 64 0.82 to 0.94; 4 for R <= 32,
//     0.86 to 0.99, but 6 for long lists of large batches (4: 1.06 at L = 500);
//   resident at 5 (20 per SM): 5.  uint8 0.95, FP32 0.96, BF16 0.98 (worst 1.03);
//   resident at 6: 6; 5 leaves queries for a second round (10k rows, 3,500 queries, L = 200:
//     uint8 1.22, FP32 1.27, BF16 1.18).  BF16 with R <= 32 in the register worklist 5, 0.96;
//   more, register worklist: uint8 7 (L = 64 0.96, two parents per hop 0.99), 8 for L <= 32
//     (0.97, worst 1.03; two parents per hop 1.02, worst 1.08); FP32 and BF16 7 is 1.01 (worst
//     1.06), so 6;
//   more, shared-memory worklist: L > 256 6 (7: uint8 1.12, FP32 1.05: no L1 left); searches
//     of builds 7, 0.98; resident at 7 (28 per SM) 7, 0.96 (worst 1.10; with R <= 32 1.02 to
//     1.04, so 6); FP32 above 36 per SM 7, 0.99; else 6 (uint8 with 7, L = 200: 1.06), BF16 6
//     throughout (7: 1.11 to 1.2).
inline int search_variant(const SearchShape& s, int sms) {
    constexpr int kF32 = 0, kBF16 = 1, kFP8 = 2, kU8 = 3;
    if (s.D > 128 || s.R > 64 || s.store > kU8) return kBlocks6;  // the only one compiled, or PQ
    const uint64_t n = s.nq, m = (uint64_t)sms;
    const bool     reg = s.L <= 64, short_list = s.R <= 32;
    if (n <= 16 * m) return kBlocks4;
    if (s.store == kFP8) return !short_list ? kBlocks5 : (n > 36 * m && s.L > 256 ? kBlocks6 : kBlocks4);
    if (n <= 20 * m) return kBlocks5;
    if (n <= 24 * m) return reg && short_list && s.store == kBF16 ? kBlocks5 : kBlocks6;
    if (s.store == kBF16) return kBlocks6;
    if (reg) {
        if (s.store == kF32 || (short_list && n <= 36 * m)) return kBlocks6;
        return s.L <= 32 && s.beam != 2 ? kBlocks8 : kBlocks7;
    }
    if (s.L > 256) return kBlocks6;
    if (s.int_queries) return kBlocks7;
    if (n <= 28 * m) return short_list ? kBlocks6 : kBlocks7;
    return s.store == kF32 && n > 36 * m ? kBlocks7 : kBlocks6;
}

}  // namespace vann
