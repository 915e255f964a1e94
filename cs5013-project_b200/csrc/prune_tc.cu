// prune_tc.cu -- RobustPrune with the candidates' Gram matrix on the tensor cores.
//
// Same decisions as prune_kernel (prune.cu), which restates pruneOutNeighbors /
// pruneReverseEdges (vamana/include/kernels.cuh:232-356, 626-743), for indexes
// whose rows are integers in [0, 255] held exactly in the uint8 copy.  For such
// rows every squared distance is an integer below 2^24 when D <= 256, so FP32
// sums in any order, and the integer identity |x|^2 + |y|^2 - 2 x.y, give the
// same value: the decisions are bit-identical to the FP32 path.
//
// One CTA (4 warps for the 128 TMEM lanes, 8 in the larger classes) prunes one node at a
// time:
//   1. candidate ids (A then B, as in prune.cu) with their distances to the node
//      (given by the search, or computed exactly from the uint8 rows);
//   2. stable order by (distance, candidate index): a candidate's rank is the count of
//      the distances below its own, equal ones of lower index included;
//   3. the first `cap` candidates' uint8 rows are staged in shared memory in that
//      order, in the K-major no-swizzle layout tcgen05.mma reads (8-row x 16-byte
//      core matrices), and one thread issues tcgen05.mma.kind::i8 (u8 x u8 -> s32)
//      for the Gram matrix G = C C^T into tensor memory (TMEM), tile by tile;
//   4. thread t reads TMEM lane t (row t of G, which is its column t) and writes the
//      bits of the earlier candidates u that, once chosen, prune t: alpha * d(u, t) <=
//      d(node, t).  Only the tiles on and below the diagonal are computed;
//   5. one warp decides the candidates on those bits, 32 at a time: a candidate is out
//      when a chosen one of an earlier word prunes it; within the word every candidate
//      with no undecided pruner is chosen, what those prune is out, and so on (a few
//      rounds of two ballots, where one p* after the other took a shuffle each);
//   6. all threads write the list and its filter slots.
// The phases are short dependent chains (loads, barriers, ballots), so what bounds the
// kernel is how many nodes an SM has in flight: up to 128 candidates a CTA takes 64
// TMEM columns and fits 8 times (tiles of 128 x 64), larger classes 128 columns, 4 at
// most.  Nodes with more candidates than a pass holds go to the next pass (256, 512,
// 768), larger ones to prune_kernel.  The host takes these passes only when it has read
// that the uint8 copy is exact; the device flag is checked again as a safeguard, and a
// kernel that finds it set hands every node on.
//
// Float rows (F16, D <= 128): the tensor cores are a filter, the decisions stay those of
// FP32.  The rows are staged relative to the node, scaled by a power of two and rounded
// to f16 (kind::f16, FP32 accumulators); a pair whose test is farther from equality than
// the rounding can move it (a bound proven beside the test, 0.22% of d(node, t)) is
// decided from the Gram entry.  The others, around 1% of the pairs, are listed and
// decided by their FP32 distance, summed in the order the warp-per-node kernel sums it,
// so every list has the bits prune_kernel gives.  A node with more undecided pairs than
// the list holds goes to the next pass, at last to prune_kernel.  f16 and not tf32: the
// same 11-bit significand (the scaling takes care of the range) at half the shared memory,
// which is what limits the nodes in flight.  prune_kernel does a node's distances on the
// CUDA cores from L2, 12 warps per SM: 42.2 ms of a 100k x 96 build's 58.7 ms.
#include <cuda_fp16.h>

#include "common.cuh"
#include "kernels.h"

namespace vann {
namespace {

// Threads of a CTA: 4 warps (the 128 TMEM lanes) for the smallest class, whose nodes in
// flight fill the SM; 8 for the larger ones, where few CTAs fit and each phase's length
// counts (two warps share a quarter of the lanes and split the columns).
__host__ __device__ constexpr uint32_t tc_threads(uint32_t maxc) { return maxc == 128u ? 128u : 256u; }
constexpr uint32_t kMaxR     = 128;
constexpr long long kSpinCycles = 2000000000ll;  // ~1 s bound on an MMA completion wait

__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor: K-major, no swizzle; lbo = byte distance
// between the two 16-byte K chunks of one MMA, sbo = between 8-row groups
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// instruction descriptor, A and B K-major and of one type: unsigned 8-bit into s32, or
// f16 into f32
template <bool F16>
__device__ __forceinline__ uint32_t idesc(uint32_t M, uint32_t N) {
    return ((F16 ? 1u : 2u) << 4) | ((N >> 3) << 17) | ((M >> 4) << 24);
}

template <bool F16>
__device__ __forceinline__ void mma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t desc, uint32_t accumulate) {
    if constexpr (F16)
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
            "l"(da), "l"(db), "r"(desc), "r"(accumulate)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
            "l"(da), "l"(db), "r"(desc), "r"(accumulate)
            : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 16 consecutive columns of this thread's TMEM lane; the wait is in the same asm
// statement so no use of r can be scheduled before the data has arrived
__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
          "=r"(r[15])
        : "r"(addr)
        : "memory");
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// bounded wait for the MMA commit of the given phase
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    const long long t0 = clock64();
    while (!mbar_try(bar, parity))
        if (clock64() - t0 > kSpinCycles) return false;
    return true;
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ uint32_t dp4a_u(uint32_t a, uint32_t b, uint32_t c) { return __dp4a(a, b, c); }

// Bytes of a staged row: D uint8, or D f16 padded to the MMA's K of 16.
__host__ __device__ constexpr uint32_t staged_bytes(uint32_t D, bool f16) {
    return f16 ? 2u * ((D + 15u) & ~15u) : D;
}

// shared memory of one CTA handling up to maxc candidates per node
struct TcLayout {
    uint32_t rows, nodev, cid, cd, sid, sd, nrm, pby, bmask, chosen, pairs, bar, misc, bytes;
    __host__ __device__ static TcLayout make(uint32_t D, uint32_t maxc, bool f16) {
        TcLayout l;
        l.rows   = 0;  // maxc staged rows, canonical layout, sorted order
        l.nodev  = l.rows + maxc * staged_bytes(D, f16);  // the node's row: uint8 or FP32
        l.cid    = l.nodev + ((f16 ? 4u * D : D) + 15u & ~15u);
        l.cd     = l.cid + 4 * maxc;  // candidate order (A then B)
        l.sid    = l.cd + 4 * maxc;   // sorted order: id (top bit: a B candidate), distance,
        l.sd     = l.sid + 4 * maxc;  // squared norm (uint8 rows)
        l.nrm    = l.sd + 4 * maxc;
        l.pby    = l.nrm + (f16 ? 0u : 4 * maxc);  // [maxc / 32][maxc] bits of the candidates that prune t
        l.bmask  = l.pby + maxc * maxc / 8;        // sorted positions holding B candidates
        l.chosen = l.bmask + 4 * ((maxc + 255u) / 256u * 8u);  // the node's new list
        l.pairs  = l.chosen + 4 * kMaxR;                               // undecided pairs (f16 rows)
        l.bar    = l.pairs + (f16 ? 4 * kPairs(maxc) : 0u);
        l.misc   = l.bar + 8;
        l.bytes  = l.misc + 4 * 16;
        return l;
    }
    // undecided pairs a node may have; one with more goes to the next pass
    __host__ __device__ static constexpr uint32_t kPairs(uint32_t maxc) { return maxc > 512u ? 2048u : 4u * maxc; }
};

// FP32 squared distance of rows x and y by a half warp (lane t of 16), in the order of
// dist_group<StoreF32> in the D <= 128 class: 8 dimensions per lane, even and odd
// apart, then the lanes pairwise (^ 8, 4, 2, 1).
__device__ __forceinline__ float half_warp_dist(const float* x, const float* y, uint32_t D, uint32_t t) {
    const float2 neg1 = make_float2(-1.f, -1.f);
    float2       acc  = make_float2(0.f, 0.f);
#pragma unroll
    for (uint32_t c = 0; c < 2; ++c) {
        const uint32_t d0 = 8u * t + 4u * c;
        if (d0 < D) {
            const float4 a = __ldg(reinterpret_cast<const float4*>(x + d0));
            const float4 b = __ldg(reinterpret_cast<const float4*>(y + d0));
            float2       d = __ffma2_rn(make_float2(a.x, a.y), neg1, make_float2(b.x, b.y));
            acc            = __ffma2_rn(d, d, acc);
            d              = __ffma2_rn(make_float2(a.z, a.w), neg1, make_float2(b.z, b.w));
            acc            = __ffma2_rn(d, d, acc);
        }
    }
    float v = acc.x + acc.y;
#pragma unroll
    for (int o = 8; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Nodes are the slots in_list[0 .. *in_count) (or 0 .. n_nodes when in_list is
// null); nodes with more than MAXC candidates go to out_list.  COLS: TMEM columns per
// CTA, the width of a Gram tile.  F16: float rows (the filter described above).
template <uint32_t MAXC, uint32_t COLS, bool F16>
__global__ void __launch_bounds__(tc_threads(MAXC), MAXC == 128 ? 8 : (MAXC == 256 ? (F16 ? 2 : 4) : 1))
    prune_tc_kernel(PruneArgs a, uint32_t* counter, const uint32_t* in_list, const uint32_t* in_count,
                    uint32_t* out_list, uint32_t* out_count) {
    constexpr uint32_t kThreads = tc_threads(MAXC);
    constexpr uint32_t kSplit   = kThreads / 128;                    // warps per quarter of the TMEM lanes
    constexpr uint32_t KPT      = (MAXC + kThreads - 1) / kThreads;  // candidates per thread
    constexpr uint32_t kB       = 0x80000000u;                       // sid: a B candidate (ids are below 2^31)
    extern __shared__ __align__(1024) unsigned char smem[];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint64_t nwork = in_list ? (uint64_t)*reinterpret_cast<volatile const uint32_t*>(in_count) : a.n_nodes;
    if (nwork == 0) return;
    if (!F16 && *reinterpret_cast<volatile const uint32_t*>(a.gate) != 0u) {  // rows not exact: hand every node on
        for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + tid; i < nwork; i += (uint64_t)gridDim.x * blockDim.x)
            out_list[atomicAdd(out_count, 1u)] = in_list ? __ldg(in_list + i) : (uint32_t)i;
        return;
    }

    const uint32_t D = a.D, R = a.R;
    const TcLayout lay = TcLayout::make(D, MAXC, F16);
    unsigned char* rows   = smem + lay.rows;
    uint8_t*       nodev  = smem + lay.nodev;
    uint32_t*      cid    = reinterpret_cast<uint32_t*>(smem + lay.cid);
    float*         cd     = reinterpret_cast<float*>(smem + lay.cd);
    uint32_t*      sid    = reinterpret_cast<uint32_t*>(smem + lay.sid);
    float*         sd     = reinterpret_cast<float*>(smem + lay.sd);
    uint32_t*      nrm    = reinterpret_cast<uint32_t*>(smem + lay.nrm);
    uint32_t*      pby    = reinterpret_cast<uint32_t*>(smem + lay.pby);
    uint32_t*      bmask  = reinterpret_cast<uint32_t*>(smem + lay.bmask);
    uint32_t*      chosen = reinterpret_cast<uint32_t*>(smem + lay.chosen);
    uint32_t*      pairs  = reinterpret_cast<uint32_t*>(smem + lay.pairs);
    // [0] tmem, [1] degree, [2..13] work items, [14] undecided pairs
    uint32_t*      misc   = reinterpret_cast<uint32_t*>(smem + lay.misc);
    const uint32_t bar    = saddr(smem + lay.bar);
    const uint32_t rows_s = saddr(rows);

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(misc)),
                     "r"(COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = misc[0];

    const bool     rev    = a.csr_off != nullptr;
    const uint32_t RB     = staged_bytes(D, F16);
    const uint32_t nchunk = RB / 16;  // 16-byte chunks of a staged row
    const uint32_t inv_nc = 0xFFFFFFFFu / nchunk + 1u;  // x / nchunk = __umulhi(x, inv_nc), nchunk >= 2
    const uint32_t LBO = 128, SBO = 8 * RB;  // 8 rows x 16 B per core matrix; chunks adjacent
    const uint32_t ksteps = RB / 32;        // K = 32 (kind::i8) or 16 (kind::f16) per instruction
    uint32_t       phase  = 0;
    bool           failed = false;
    uint32_t       done   = 0;  // nodes pruned by this CTA

    // The next work item (slot, node, |A|, A offset, |B|) is fetched by one thread
    // while the CTA prunes the current one, so its chain of dependent loads (work
    // counter, node id, list bounds, degree) is off the critical path.
    auto fetch = [&](uint32_t* item) {
        uint32_t       w = kNone, node = kNone, nA = 0, aoff = 0, nB = 0;
        const uint32_t i = atomicAdd(counter, 1u);
        if (i < nwork) {
            w    = in_list ? __ldg(in_list + i) : i;
            node = a.node_ids ? __ldg(a.node_ids + w) : w;  // kNone: the padded slots' run
            if (node != kNone) {
                if (rev) {
                    const uint32_t ci = a.csr_by_slot ? w : node;
                    nA                = __ldg(a.csr_cnt + ci);
                    aoff              = __ldg(a.csr_off + ci);
                    if (a.skip_empty && nA == 0u) node = kNone;
                    nA = min(nA, a.cap);
                } else {
                    nA = min(__ldg(a.a_n + w), a.a_stride);
                }
                if (node != kNone && a.use_b) nB = min(a.deg[node], R);
            }
        }
        item[0] = w;
        item[1] = node;
        item[2] = nA;
        item[3] = aoff;
        item[4] = nB;
    };
    if (tid == 32) fetch(misc + 2);
    __syncthreads();

    for (uint32_t it = 0;; ++it, __syncthreads()) {
        const uint32_t* cur  = misc + 2 + 6 * (it & 1u);
        const uint32_t  w    = cur[0];
        const uint32_t  node = cur[1];
        const uint32_t  nA = cur[2], aoff = cur[3], nB = cur[4];
        if (w == kNone) break;
        if (tid == 32) fetch(misc + 2 + 6 * ((it + 1u) & 1u));
        if (node == kNone) continue;
        const uint32_t nc = nA + nB;
        if (nc > MAXC) {
            if (tid == 0) out_list[atomicAdd(out_count, 1u)] = w;
            continue;
        }
        const bool computed = rev || nB > 0 || a.a_d == nullptr;  // some distance is not given

        // --- 1. candidate ids (A then B) and given distances; the node's row
        for (uint32_t i = tid; i < nc; i += kThreads) {
            uint32_t id;
            float    d = -1.f;  // computed below
            if (i < nA) {
                if (rev) {
                    id = __ldg(a.csr_src + aoff + i);
                } else {
                    id = __ldg(a.a_ids + (uint64_t)w * a.a_stride + i);
                    if (a.a_d) d = __ldg(a.a_d + (uint64_t)w * a.a_stride + i);
                }
            } else {
                id = __ldg(a.adj + (uint64_t)node * R + (i - nA));
            }
            cid[i] = id;
            cd[i]  = d;
        }
        if (tid < 32u && ((nc + 31u) & ~31u) > nc + tid)  // the last chunk of 32 is read whole below
            cd[nc + tid] = __uint_as_float(0xFFFFFFFFu);
        if constexpr (F16) {
            if (tid < D / 4u)
                reinterpret_cast<float4*>(nodev)[tid] =
                    __ldg(reinterpret_cast<const float4*>(a.vecs + (uint64_t)node * D) + tid);
            const uint32_t first = (rev || a.a_d == nullptr) ? 0u : nA;
            if (first < nc) {  // missing distances from the FP32 rows, as the search takes them
                constexpr uint32_t G = Layout<StoreF32, 0>::kG;
                __syncthreads();
                Query<StoreF32, 0> nv;
                load_query<StoreF32, 0>(nv, a.vecs + (uint64_t)node * D, D, lane);
                for (uint32_t g0 = first + warp * G; g0 < nc; g0 += G * (kThreads / 32u))
                    dist_round<StoreF32, 0>(nv, a.vecs, nullptr, [&](int j) { return cid[g0 + j]; },
                                            (int)min(G, nc - g0), D, lane, cd + g0);
            }
        } else if (computed) {
            if (tid < nchunk)
                *reinterpret_cast<uint4*>(nodev + 16 * tid) =
                    __ldg(reinterpret_cast<const uint4*>(a.vecs_u8 + (uint64_t)node * D) + tid);
            __syncthreads();
            // missing distances straight from the uint8 rows (exact integers)
            uint32_t nn = 0;  // |node|^2
            for (uint32_t c = 0; c < nchunk; ++c) {
                const uint4 q = *reinterpret_cast<const uint4*>(nodev + 16 * c);
                nn = dp4a_u(q.x, q.x, dp4a_u(q.y, q.y, dp4a_u(q.z, q.z, dp4a_u(q.w, q.w, nn))));
            }
            for (uint32_t i = tid; i < nc; i += kThreads) {
                if (cd[i] >= 0.f) continue;
                const uint4* row = reinterpret_cast<const uint4*>(a.vecs_u8 + (uint64_t)cid[i] * D);
                uint32_t     n = 0, dot = 0;
                for (uint32_t c = 0; c < nchunk; ++c) {
                    const uint4 v = __ldg(row + c);
                    const uint4 q = *reinterpret_cast<const uint4*>(nodev + 16 * c);
                    n   = dp4a_u(v.x, v.x, dp4a_u(v.y, v.y, dp4a_u(v.z, v.z, dp4a_u(v.w, v.w, n))));
                    dot = dp4a_u(v.x, q.x, dp4a_u(v.y, q.y, dp4a_u(v.z, q.z, dp4a_u(v.w, q.w, dot))));
                }
                cd[i] = (float)(nn + n - 2u * dot);
            }
        }
        __syncthreads();

        // --- 2. stable order by (distance, candidate index).  Distances are non-negative,
        // so their bits order them: rank = distances below, plus equal ones of lower index
        // (whole chunks of 32 by a raised bound, the candidate's own chunk by a match).
        const uint32_t m = min(nc, a.cap);
        {
            uint32_t b[KPT], r[KPT];
#pragma unroll
            for (uint32_t q = 0; q < KPT; ++q) {
                const uint32_t i = tid + q * kThreads;
                b[q]             = i < nc ? __float_as_uint(cd[i]) : 0u;
                r[q]             = __popc(__match_any_sync(0xffffffffu, b[q]) & ((1u << lane) - 1u));
            }
            const uint32_t used = (nc + kThreads - 1) / kThreads;  // candidates in use per thread
            for (uint32_t c0 = 0; c0 < nc; c0 += 32) {  // the warp's own chunk: kThreads q + 32 warp
                const uint4* dj = reinterpret_cast<const uint4*>(cd + c0);
                uint32_t     thr[KPT];
#pragma unroll
                for (uint32_t q = 0; q < KPT; ++q) thr[q] = b[q] + (c0 < kThreads * q + 32u * warp ? 1u : 0u);
#pragma unroll
                for (uint32_t j = 0; j < 8; ++j) {
                    const uint4 x = dj[j];
#pragma unroll
                    for (uint32_t q = 0; q < KPT; ++q)
                        if (q < used)
                            r[q] += (uint32_t)(x.x < thr[q]) + (uint32_t)(x.y < thr[q]) + (uint32_t)(x.z < thr[q]) +
                                    (uint32_t)(x.w < thr[q]);
                }
            }
#pragma unroll
            for (uint32_t q = 0; q < KPT; ++q) {
                const uint32_t i = tid + q * kThreads;
                if (i < nc && r[q] < m) {
                    sid[r[q]] = cid[i] | (i >= nA ? kB : 0u);
                    sd[r[q]]  = __uint_as_float(b[q]);
                }
            }
        }
        __syncthreads();

        // --- 3. the first `cap` candidates' rows staged for the MMA
        float g2 = 0.f, slack = 0.f;  // f16 rows: 2 / scale^2, and the error bound's constant part
        if constexpr (F16) {
            // rows relative to the node, scaled by a power of two so that the longest is
            // at most 2^14, rounded to f16
            const float smax = m > 0u ? sd[m - 1u] : 0.f;  // squared length of the longest
            const bool  sane = smax > 1e-30f && smax < 1e37f;
            int         e    = 0;
            if (sane) frexpf(smax, &e);  // smax < 2^e
            const int   h    = 14 - ((e + 1) >> 1);
            const float up   = ldexpf(1.f, h);
            g2               = ldexpf(2.f, -2 * h);
            slack            = sane ? 1e-9f * smax : __int_as_float(0x7f800000);
            const float4* nf = reinterpret_cast<const float4*>(nodev);
            if (tid == 0) misc[14] = 0u;
#pragma unroll 4
            for (uint32_t x = tid; x < m * nchunk; x += kThreads) {
                const uint32_t t = __umulhi(x, inv_nc), c = x - t * nchunk;
                const float4*  src = reinterpret_cast<const float4*>(a.vecs + (uint64_t)(sid[t] & ~kB) * D) + 2u * c;
                uint32_t       p[4] = {0u, 0u, 0u, 0u};
#pragma unroll
                for (uint32_t v = 0; v < 2; ++v) {
                    if (8u * c + 4u * v < D) {
                        const float4  r = __ldg(src + v), n = nf[2u * c + v];
                        const __half2 lo = __floats2half2_rn((r.x - n.x) * up, (r.y - n.y) * up);
                        const __half2 hi = __floats2half2_rn((r.z - n.z) * up, (r.w - n.w) * up);
                        p[2 * v]         = *reinterpret_cast<const uint32_t*>(&lo);
                        p[2 * v + 1]     = *reinterpret_cast<const uint32_t*>(&hi);
                    }
                }
                *reinterpret_cast<uint4*>(rows + (t >> 3) * SBO + c * LBO + (t & 7u) * 16u) =
                    make_uint4(p[0], p[1], p[2], p[3]);
            }
        } else {
            for (uint32_t x = tid; x < m * nchunk; x += kThreads) {
                const uint32_t t = __umulhi(x, inv_nc), c = x - t * nchunk;
                cp_async16(rows_s + (t >> 3) * SBO + c * LBO + (t & 7u) * 16u,
                           a.vecs_u8 + (uint64_t)(sid[t] & ~kB) * D + 16u * c);
            }
        }
        if (a.consistent) {
#pragma unroll
            for (uint32_t q = 0; q < KPT; ++q) {
                const uint32_t t    = kThreads * q + tid;
                const uint32_t bits = __ballot_sync(0xffffffffu, t < m && (sid[t] & kB) != 0u);
                if (lane == 0) bmask[(kThreads / 32u) * q + warp] = bits;
            }
        }
        cp_async_wait_all();
        fence_proxy_async();  // rows become visible to the tensor core's reads
        __syncthreads();

        // --- 4. Gram tiles on the tensor cores; squared norms of the staged rows
        const uint32_t nb = (m + 127u) / 128u;  // row blocks of 128
        auto issue_tile = [&](uint32_t r, uint32_t c) {
            const uint32_t left = m - COLS * c;
            const uint32_t N    = ((left < COLS ? left : COLS) + 15u) & ~15u;
            const uint32_t id   = idesc<F16>(128u, N);
            for (uint32_t s = 0; s < ksteps; ++s) {
                const uint64_t da = umma_desc(rows_s + r * 16u * SBO + s * 2u * LBO, LBO, SBO);
                const uint64_t db = umma_desc(rows_s + c * (COLS / 8u) * SBO + s * 2u * LBO, LBO, SBO);
                mma<F16>(tmem, da, db, id, s > 0 ? 1u : 0u);
            }
            mma_commit(bar);
        };
        if (m > 0 && tid == 0) {
            tc_fence_after();
            issue_tile(0, 0);
        }
        if constexpr (!F16) {
            for (uint32_t t = tid; t < m; t += kThreads) {
                uint32_t n = 0;
                for (uint32_t c = 0; c < nchunk; ++c) {
                    const uint4 v = *reinterpret_cast<const uint4*>(rows + (t >> 3) * SBO + c * LBO + (t & 7u) * 16u);
                    n = dp4a_u(v.x, v.x, dp4a_u(v.y, v.y, dp4a_u(v.z, v.z, dp4a_u(v.w, v.w, n))));
                }
                nrm[t] = n;
            }
            __syncthreads();
        }

        // --- 5. bits of the candidates that prune t.  A thread whose wait gave up neither
        // issues a tile nor waits again, and one left waiting for a tile that was not issued
        // gives up too: two bounds at most for the node, not one per tile (21 in the largest
        // class).  (A vote at each tile's barrier, or the walk as a function over lambdas,
        // made a 5% consolidation of 300k rows 10.0 -> 10.1 ms.)
        bool late = false;
        for (uint32_t r = 0; r < nb; ++r) {
            const uint32_t t = 128u * r + (tid & 127u);
            // "u prunes t" is alpha * d(u, t) <= d(node, t) in FP32, with d(u, t) the exact
            // integer Y = |u|^2 + |t|^2 - 2 u.t (< 2^24, so FP32 holds it exactly).  fl(Y *
            // alpha) does not decrease as Y grows, so the test is Y <= Ymax(t), the largest
            // integer with fl(Ymax * alpha) <= d(node, t): 2 u.t - |u|^2 >= |t|^2 - Ymax(t).
            // Float rows: with the Gram entry g of the f16 rows, d(u, t) is su + st - g2 g up
            // to an error E, so u prunes t for certain where g2 g - su > st - st / alpha + E,
            // and for certain not where it is < st - st / alpha - E (su <= st: u comes first).
            // E: f16 rounding of both rows (2^-11 of each component) and the tensor core's
            // FP32 accumulation, 2 (2^-10 + 2^-15) sqrt(su st) <= 0.00202 st; the FP32 sums
            // su, st and d(u, t) themselves and this test's arithmetic, 4e-5 st; f16
            // subnormals, 1e-9 of the longest row; FP32 subnormals, 1e-37.
            int      thr  = 0;
            float    flo = 0.f, fhi = 0.f;
            uint32_t keep = ~0u;  // consistent lists: no B candidate is checked against another
            if (t < m) {
                const float sdt = sd[t];
                if constexpr (F16) {
                    const float mid = sdt - sdt / a.alpha;
                    const float err = 0.0022f * sdt + slack + 1e-37f;
                    flo             = mid - err;
                    fhi             = mid + err;
                } else {
                    int y = (int)fminf(floorf(sdt / a.alpha), 16777215.f);
                    while (y < 16777215 && (float)(y + 1) * a.alpha <= sdt) ++y;
                    while (y > 0 && (float)y * a.alpha > sdt) --y;
                    thr = (int)nrm[t] - y;
                }
                if (a.consistent && (sid[t] & kB)) keep = 0u;
            }
            const uint32_t last  = 128u * r + 32u * (warp & 3u) + 31u;  // the warp's last candidate
            const uint32_t ncols = min(m, 128u * (r + 1u));
            for (uint32_t c = 0; COLS * c < ncols; ++c) {
                if (r != 0 || c != 0) {
                    tc_fence_before();
                    __syncthreads();  // every thread's reads of the previous tile are done
                    if (tid == 0 && !late) {
                        tc_fence_after();
                        issue_tile(r, c);
                    }
                }
                if (!late) {
                    late = !mbar_wait(bar, phase);
                    phase ^= 1u;
                }
                tc_fence_after();
#pragma unroll 1
                for (uint32_t c32 = 32u * (warp >> 2); c32 < COLS; c32 += 32u * kSplit) {
                    const uint32_t u0 = COLS * c + c32;
                    if (u0 >= m || u0 > last) break;
                    uint32_t word = 0, open = 0;  // open: undecided (float rows)
#pragma unroll
                    for (uint32_t h = 0; h < 32u; h += 16u) {
                        if (u0 + h < m) {
                            uint32_t g[16];
                            tmem_ld16(tmem + ((32u * (warp & 3u)) << 16) + c32 + h, g);
#pragma unroll
                            for (uint32_t k = 0; k < 16; k += 4) {
                                if constexpr (F16) {
                                    const float4 su  = *reinterpret_cast<const float4*>(sd + u0 + h + k);
                                    const float  x[4] = {fmaf(__uint_as_float(g[k]), g2, -su.x),
                                                         fmaf(__uint_as_float(g[k + 1]), g2, -su.y),
                                                         fmaf(__uint_as_float(g[k + 2]), g2, -su.z),
                                                         fmaf(__uint_as_float(g[k + 3]), g2, -su.w)};
#pragma unroll
                                    for (uint32_t i = 0; i < 4; ++i) {
                                        const bool yes = x[i] > fhi;
                                        word |= (uint32_t)yes << (h + k + i);
                                        open |= (uint32_t)(!yes && !(x[i] < flo)) << (h + k + i);
                                    }
                                } else {
                                    const uint4 nu = *reinterpret_cast<const uint4*>(nrm + u0 + h + k);
                                    word |= (uint32_t)((int)(2u * g[k] - nu.x) >= thr) << (h + k);
                                    word |= (uint32_t)((int)(2u * g[k + 1] - nu.y) >= thr) << (h + k + 1);
                                    word |= (uint32_t)((int)(2u * g[k + 2] - nu.z) >= thr) << (h + k + 2);
                                    word |= (uint32_t)((int)(2u * g[k + 3] - nu.w) >= thr) << (h + k + 3);
                                }
                            }
                        }
                    }
                    if (keep == 0u) word &= ~bmask[u0 >> 5];
                    if (t < m) pby[(u0 >> 5) * MAXC + t] = word;
                    if constexpr (F16) {
                        if (keep == 0u) open &= ~bmask[u0 >> 5];
                        if (u0 + 32u > t) open &= t > u0 ? (1u << (t - u0)) - 1u : 0u;  // earlier candidates only
                        if (t < m && open != 0u) {
                            uint32_t at = atomicAdd(&misc[14], __popc(open));
                            for (; open != 0u && at < TcLayout::kPairs(MAXC); open &= open - 1u, ++at)
                                pairs[at] = (t << 16) | (u0 + __ffs(open) - 1u);
                        }
                    }
                }
            }
        }
        tc_fence_before();
        if (__syncthreads_or(late)) {  // a wait for the tensor cores gave up
            // bounded: products still in flight write the tensor memory that is freed below
            if (tid == 0 && late) mbar_wait(bar, phase ^ 1u);
            failed = true;
            break;
        }

        if constexpr (F16) {
            // undecided pairs by their FP32 distance, a half warp each
            const uint32_t np = misc[14];
            if (np > TcLayout::kPairs(MAXC)) {
                if (tid == 0) out_list[atomicAdd(out_count, 1u)] = w;
                continue;
            }
            for (uint32_t p0 = 2u * warp; p0 < np; p0 += 2u * (kThreads / 32u)) {
                const uint32_t p  = p0 + (lane >> 4);
                const uint32_t pr = pairs[min(p, np - 1u)], t = pr >> 16, u = pr & 0xffffu;
                const float    y  = half_warp_dist(a.vecs + (uint64_t)(sid[u] & ~kB) * D,
                                                   a.vecs + (uint64_t)(sid[t] & ~kB) * D, D, lane & 15u);
                if ((lane & 15u) == 0u && p < np && y * a.alpha <= sd[t])
                    atomicOr(&pby[(u >> 5) * MAXC + t], 1u << (u & 31u));
            }
            __syncthreads();
        }

        // --- 6. selection (warp 0), a word of 32 candidates at a time
        if (warp == 0) {
            uint32_t       ndeg  = 0, sel = 0;  // lane q: the chosen candidates of word q
            const uint32_t words = (m + 31u) / 32u;
            for (uint32_t k = 0; k < words && ndeg < R; ++k) {
                const uint32_t t   = 32u * k + lane;
                uint32_t       out = t < m ? 0u : 1u;
                for (uint32_t q = 0; q < k; ++q) {
                    const uint32_t s = __shfl_sync(0xffffffffu, sel, q);
                    out |= pby[q * MAXC + t] & s;
                }
                const uint32_t by   = pby[k * MAXC + t] & ((1u << lane) - 1u);  // pruners within the word
                uint32_t       und  = __ballot_sync(0xffffffffu, out == 0u);
                uint32_t       got  = 0u;
                while (und != 0u) {
                    const bool     in  = (und >> lane) & 1u;
                    const uint32_t now = __ballot_sync(0xffffffffu, in && (by & und) == 0u);
                    got |= now;
                    und &= ~now & ~__ballot_sync(0xffffffffu, in && (by & now) != 0u);
                }
                const uint32_t rank = __popc(got & ((1u << lane) - 1u));
                const bool     mine = ((got >> lane) & 1u) && ndeg + rank < R;
                if (mine) chosen[ndeg + rank] = sid[t] & ~kB;
                ndeg = min(R, ndeg + __popc(got));
                if (lane == k) sel = got;
            }
            if (lane == 0) {
                misc[1]     = ndeg;
                a.deg[node] = ndeg;
            }
        }
        __syncthreads();
        // the new list and its filter slots, one entry per thread
        if (tid < misc[1]) {
            const uint32_t id                 = chosen[tid];
            a.adj[(uint64_t)node * R + tid]   = id;
            a.adj_h[(uint64_t)node * R + tid] = bloom_pack(id);
        }
        ++done;
    }
    if (failed && tid == 0) atomicOr(a.status, kStatusTimeout);
    if (tid == 0 && a.pruned && done) atomicAdd(a.pruned + (F16 ? 1 : 0), (unsigned long long)done);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS));
    }
}

}  // namespace

bool prune_tc_supported(uint32_t D, uint32_t R) { return D % 32 == 0 && D >= 32 && D <= 256 && R <= kMaxR; }
bool prune_f16_supported(uint32_t D, uint32_t R) { return D <= 128 && R <= kMaxR; }

namespace {

template <uint32_t MAXC, uint32_t COLS, bool F16 = false>
cudaError_t launch_tc(const PruneArgs& a, uint32_t* counter, const uint32_t* in_list, const uint32_t* in_count,
                      uint32_t* out_list, uint32_t* out_count, uint64_t max_nodes, int num_sms, cudaStream_t st) {
    int dev = 0, per_sm_smem = 0, reserved = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&per_sm_smem, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev);
    if (e != cudaSuccess) return e;
    // TMEM holds 512 columns per SM: at most 512 / COLS CTAs of these kernels may
    // share an SM, which the shared-memory request enforces (an extra CTA would wait
    // in tcgen05.alloc for one of the others to exit).
    const int    max_ctas    = 512 / (int)COLS;
    size_t       smem        = TcLayout::make(a.D, MAXC, F16).bytes;
    const size_t floor_bytes = (size_t)(per_sm_smem / (max_ctas + 1) - reserved + 1024);
    if (smem < floor_bytes) smem = floor_bytes;
    auto kern = prune_tc_kernel<MAXC, COLS, F16>;
    e = allow_smem(kern, smem);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                             (int)cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    // CTAs per SM from the shared-memory budget (the occupancy query reports one CTA
    // per SM for kernels that allocate tensor memory, which is not the limit here)
    int per_sm = per_sm_smem / (int)(smem + reserved);
    if (per_sm > max_ctas) per_sm = max_ctas;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    uint64_t grid = (uint64_t)per_sm * num_sms;
    if (grid > max_nodes) grid = max_nodes;
    kern<<<(unsigned)grid, tc_threads(MAXC), smem, st>>>(a, counter, in_list, in_count, out_list, out_count);
    return cudaGetLastError();
}

}  // namespace

// Passes of 128 candidates (up to 8 CTAs per SM), 256 (4), 512 (2), then 768 (one per
// SM, when its shared memory fits: D <= 160), each over the nodes the previous one
// handed on.  The first pass takes in_list[0 .. *in_count) (every node when null);
// what the last cannot take goes to out_list for prune_kernel.  A launch of no more
// nodes than SMs has nothing to fill with small passes and goes straight to the last; one
// of no more than the 256 class holds at once (4 per SM) takes that and the last.
// ws: 2 * n_nodes words of device scratch; counters, counts, out_count: zeroed.
cudaError_t launch_prune_tc(const PruneArgs& a, const uint32_t* in_list, const uint32_t* in_count,
                            uint32_t* out_list, uint32_t* out_count, uint32_t* ws, uint32_t* counters,
                            uint32_t* counts, int num_sms, cudaStream_t st) {
    if (a.n_nodes == 0) return cudaSuccess;
    if (!prune_tc_supported(a.D, a.R) || !a.vecs_u8 || !a.gate || !out_list || !out_count)
        return cudaErrorInvalidValue;
    int dev = 0, max_optin = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    const uint64_t n       = a.n_nodes;
    const bool     last768 = TcLayout::make(a.D, 768, false).bytes <= (uint32_t)max_optin;
    uint32_t*      list[2] = {ws, ws + n};
    if (last768 && n <= (uint64_t)num_sms)
        return launch_tc<768, 128>(a, counters, in_list, in_count, out_list, out_count, n, num_sms, st);
    if (last768 && n <= 4ull * (uint64_t)num_sms) {
        e = launch_tc<256, 128>(a, counters, in_list, in_count, list[0], counts, n, num_sms, st);
        if (e != cudaSuccess) return e;
        return launch_tc<768, 128>(a, counters + 1, list[0], counts, out_list, out_count, n, num_sms, st);
    }
    e = launch_tc<128, 64>(a, counters, in_list, in_count, list[0], counts, n, num_sms, st);
    if (e != cudaSuccess) return e;
    e = launch_tc<256, 128>(a, counters + 1, list[0], counts, list[1], counts + 1, n, num_sms, st);
    if (e != cudaSuccess) return e;
    if (!last768)
        return launch_tc<512, 128>(a, counters + 2, list[1], counts + 1, out_list, out_count, n, num_sms, st);
    e = launch_tc<512, 128>(a, counters + 2, list[1], counts + 1, list[0], counts + 2, n, num_sms, st);
    if (e != cudaSuccess) return e;
    return launch_tc<768, 128>(a, counters + 3, list[0], counts + 2, out_list, out_count, n, num_sms, st);
}

// The same over float rows (also exact byte rows of a length the integer passes do not
// take): passes of 128, 256 and 576 candidates.  The 256-candidate class is resident twice per
// SM here, but 2 to 4 nodes per SM are still better off without the 128-candidate pass: an
// insert of 300 to 450 rows into 100k x 96 takes 0.54 ms, 0.56 with it; x 128 0.62 and 0.64.
cudaError_t launch_prune_f16(const PruneArgs& a, const uint32_t* in_list, const uint32_t* in_count,
                             uint32_t* out_list, uint32_t* out_count, uint32_t* ws, uint32_t* counters,
                             uint32_t* counts, int num_sms, cudaStream_t st) {
    if (a.n_nodes == 0) return cudaSuccess;
    if (!prune_f16_supported(a.D, a.R) || !out_list || !out_count) return cudaErrorInvalidValue;
    const uint64_t n       = a.n_nodes;
    uint32_t*      list[2] = {ws, ws + n};
    if (n <= (uint64_t)num_sms)
        return launch_tc<576, 128, true>(a, counters, in_list, in_count, out_list, out_count, n, num_sms, st);
    cudaError_t     e   = cudaSuccess;
    const uint32_t *il = in_list, *ic = in_count;
    if (n > 4ull * (uint64_t)num_sms) {
        e  = launch_tc<128, 64, true>(a, counters, il, ic, list[0], counts, n, num_sms, st);
        il = list[0];
        ic = counts;
        if (e != cudaSuccess) return e;
    }
    e = launch_tc<256, 128, true>(a, counters + 1, il, ic, list[1], counts + 1, n, num_sms, st);
    if (e != cudaSuccess) return e;
    return launch_tc<576, 128, true>(a, counters + 2, list[1], counts + 1, out_list, out_count, n, num_sms, st);
}

}  // namespace vann
