// search_dispatch.cuh -- picks the search kernel instantiation for a launch:
// register worklist (search_reg.cuh) for L <= 64 at D <= 128 and R <= 64,
// shared-memory worklist (search_impl.cuh) otherwise, a CTA per query (search_cta.cuh)
// for small batches of either, and the launch-bound variant chosen by the autotuner.
#pragma once
#include "search_cta.cuh"
#include "search_reg.cuh"

namespace vann {

// Launch-bound variants (minimum resident blocks per SM, i.e. a register cap)
// exist for the common shape (D <= 128, R <= 64); the autotuner picks one.
constexpr int kSearchVariants = 7;

template <typename S, int DC, int SPL, int LREG, int BEAM>
static cudaError_t launch_rw_v(const SearchArgs& a, int variant, int sms, cudaStream_t st) {
    switch (variant) {
        case 1: return launch_rw<S, DC, SPL, LREG, 4, BEAM>(a, sms, st);
        case 2: return launch_rw<S, DC, SPL, LREG, 5, BEAM>(a, sms, st);
        case 3: return launch_rw<S, DC, SPL, LREG, 7, BEAM>(a, sms, st);
        case 4: return launch_rw<S, DC, SPL, LREG, 8, BEAM>(a, sms, st);
        case 5: return launch_rw<S, DC, SPL, LREG, 9, BEAM>(a, sms, st);
        case 6: return launch_rw<S, DC, SPL, LREG, 10, BEAM>(a, sms, st);
        default: return launch_rw<S, DC, SPL, LREG, 6, BEAM>(a, sms, st);
    }
}

template <typename S, int DC, int SPL>
static cudaError_t launch_v(const SearchArgs& a, int variant, int sms, cudaStream_t st) {
    if constexpr (DC == 0 && SPL <= 2) {
        // worklist in registers for L <= 64; two parents per hop only here
        if (a.L <= 32)
            return a.beam == 2 ? launch_rw_v<S, DC, SPL, 1, 2>(a, variant, sms, st)
                               : launch_rw_v<S, DC, SPL, 1, 1>(a, variant, sms, st);
        if (a.L <= 64)
            return a.beam == 2 ? launch_rw_v<S, DC, SPL, 2, 2>(a, variant, sms, st)
                               : launch_rw_v<S, DC, SPL, 2, 1>(a, variant, sms, st);
    }
    if (a.beam == 2) return cudaErrorInvalidValue;
    if constexpr (S::kInt && DC == 0 && SPL <= 2) {
        if (a.int_queries) {  // build and insert searches over the exact uint8 copy
            switch (variant) {
                case 1: return launch_t<S, DC, SPL, 4, true>(a, sms, st);
                case 2: return launch_t<S, DC, SPL, 5, true>(a, sms, st);
                case 3: return launch_t<S, DC, SPL, 7, true>(a, sms, st);
                case 4: return launch_t<S, DC, SPL, 8, true>(a, sms, st);
                case 5: return launch_t<S, DC, SPL, 9, true>(a, sms, st);
                case 6: return launch_t<S, DC, SPL, 10, true>(a, sms, st);
                default: return launch_t<S, DC, SPL, 6, true>(a, sms, st);
            }
        }
    }
    if constexpr (DC == 0 && SPL <= 2) {
        switch (variant) {
            case 1: return launch_t<S, DC, SPL, 4>(a, sms, st);
            case 2: return launch_t<S, DC, SPL, 5>(a, sms, st);
            case 3: return launch_t<S, DC, SPL, 7>(a, sms, st);
            case 4: return launch_t<S, DC, SPL, 8>(a, sms, st);
            case 5: return launch_t<S, DC, SPL, 9>(a, sms, st);
            case 6: return launch_t<S, DC, SPL, 10>(a, sms, st);
            default: break;
        }
    }
    return launch_t<S, DC, SPL, 6>(a, sms, st);
}

template <typename S, int DC>
static cudaError_t launch_r(const SearchArgs& a, int variant, int sms, cudaStream_t st) {
    if (a.R <= 32) return launch_v<S, DC, 1>(a, variant, sms, st);
    if (a.R <= 64) return launch_v<S, DC, 2>(a, variant, sms, st);
    return launch_v<S, DC, 4>(a, variant, sms, st);
}

// Batches served by a CTA per query (search_cta.cuh): up to as many queries as keep it
// ahead of a warp per query, which needs many to fill the chip but then does more of them.
// Measured on 148 SMs, CTA / warp per query in us:
//   worklist in registers otherwise (L <= 64): uint8 1M x 128, L = 64: 1 query 88 / 114, 300
//     queries 247 / 305, 590 322 / 373; uint8 L = 32: 1 query 50 / 58, 590 114 / 134 (with 8
//     rows a round instead of 4, 700 queries took 148 / 135);
//   L <= 128, or wider rows or lists: FP32 200k x 96, L = 100: 1 query 116 / 211, 590 298 /
//     479, 1,000 365 / 481 (1,200: 494 / 476); BF16 100k x 256, L = 128 with rerank: 1 query
//     242 / 493, 590 563 / 981, 1,000 837 / 1,074 (1,200: 1,126 / 1,110);
//   L <= 256 (more registers, fewer CTAs): FP32 L = 200: 1 query 189 / 319, 300 239 / 416 (590:
//     451 / 429).
inline bool small_batch(const SearchArgs& a, int sms) {
    if (a.beam == 2 || a.L > kCtaMaxL) return false;
    const uint64_t per_sm = a.L > 128 ? 3 : (a.L > 64 || a.D > 128 || a.R > 64 ? 7 : 4);
    return a.nq <= per_sm * (uint64_t)sms;
}

// Launch-bound variant (blocks of 4 warps per SM) of a search that was not autotuned.  A
// register cap trades resident warps for spills, so the choice depends on the row
// format's registers and on how many warps the batch can fill: while every query fits
// at once more registers cost nothing.  Measured, ms at 6 blocks against the choice:
//   every query resident at 4 blocks (16 queries per SM): 4.  1,800 queries: uint8 L = 58
//     0.176 / 0.167, FP8 L = 58 0.356 / 0.297, FP32 L = 120 0.677 / 0.647, BF16 0.678 / 0.632;
//   FP8 otherwise (its conversions need the registers): 4 for R <= 32, else 5.  10k on 1M x
//     128: L = 64 1.267 / 1.130, L = 100 2.290 / 1.884;
//   up to 24 per SM: 5, 6 for R <= 32 (BF16 5).  3,000 on 1M x 128: uint8 L = 64 0.458 / 0.439,
//     BF16 L = 32 0.386 / 0.373; 3,400, R = 48: uint8 L = 120 0.703 / 0.636;
//   up to 36: register worklist 6 (uint8 with R > 32: 5, 0.341 / 0.318), else as below;
//   more, register worklist: uint8 8 (10k on 1M: L = 32 0.472 / 0.458, 1M x 96 L = 64 0.750 /
//     0.716), FP32 7 for R > 32 (0.831 / 0.800; 10k rows 0.375 / 0.388), BF16 7 for L <= 32 or
//     R <= 32 (0.687 / 0.676, 0.872 / 0.844);
//   more, shared-memory worklist: uint8 and FP32 7 (uint8 L = 100 1.217 / 1.173, FP32 L = 199 on
//     10k rows 1.562 / 1.538; 8 spills: 1.406, 1.832), BF16 6.
template <typename S>
static int default_variant(const SearchArgs& a, int sms) {
    constexpr int  k4 = 1, k5 = 2, k6 = 0, k7 = 3, k8 = 4;
    constexpr bool f32 = !S::kInt && S::kElems == 4, bf16 = S::kElems == 8;
    const uint64_t n = a.nq, m = (uint64_t)sms;
    const bool     reg = a.L <= 64 && a.R <= 64, short_list = a.R <= 32;
    if (S::kPQ) return k6;
    if (n <= 16 * m) return k4;
    if (S::kScaled) return short_list ? k4 : k5;
    if (n <= 24 * m) return short_list && !(bf16 && reg) ? k6 : k5;
    if (!reg) return S::kInt || f32 ? k7 : k6;
    if (n <= 36 * m) return S::kInt && !short_list ? k5 : k6;
    if (S::kInt) return k8;
    if (f32) return short_list ? k6 : k7;
    return a.L <= 32 || short_list ? k7 : k6;
}

template <typename S>
static cudaError_t launch_store(const SearchArgs& a, int variant, int sms, cudaStream_t st) {
    if (a.D % S::kElems != 0) return cudaErrorInvalidValue;
    if constexpr (!S::kPQ) {
        if (small_batch(a, sms)) {
            if constexpr (S::kInt)
                if (a.int_queries && a.D <= 128) return launch_cta<S, 0, true>(a, sms, st);
            if (a.D <= 128) return launch_cta<S, 0>(a, sms, st);
            if (a.D <= 256) return launch_cta<S, 1>(a, sms, st);
            return launch_cta<S, 2>(a, sms, st);
        }
    }
    if (variant < 0) variant = default_variant<S>(a, sms);
    if (a.D <= 128) return launch_r<S, 0>(a, variant, sms, st);
    if (a.D <= 256) return launch_r<S, 1>(a, variant, sms, st);
    return launch_r<S, 2>(a, variant, sms, st);
}

}  // namespace vann
