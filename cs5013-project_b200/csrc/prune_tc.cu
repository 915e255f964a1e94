// prune_tc.cu -- RobustPrune with the candidates' Gram matrix on the tensor cores.
//
// Same decisions as prune_kernel (prune.cu), which restates pruneOutNeighbors /
// pruneReverseEdges (vamana/include/kernels.cuh:232-356, 626-743), for indexes
// whose rows are integers in [0, 255] held exactly in the uint8 copy.  For such
// rows every squared distance is an integer below 2^24 when D <= 256, so FP32
// sums in any order, and the integer identity |x|^2 + |y|^2 - 2 x.y, give the
// same value: the decisions are bit-identical to the FP32 path.
//
// One CTA of 4 warps (the 128 TMEM lanes) prunes one node at a time:
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
// 768), larger ones to prune_kernel.  If the uint8 copy is not exact (a device flag
// written by the conversion kernels) this kernel returns at once and prune_kernel does
// all.
#include "common.cuh"
#include "kernels.h"

namespace vann {
namespace {

constexpr uint32_t kThreads  = 128;  // 4 warps = the 128 TMEM lanes
constexpr uint32_t kMaxR     = 128;
constexpr long long kSpinCycles = 2000000000ll;  // ~1 s bound on an MMA completion wait

__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor: K-major, no swizzle; lbo = byte distance
// between the two 16-byte K chunks of one MMA, sbo = between 8-row groups
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// instruction descriptor: D s32, A and B unsigned 8-bit, both K-major
__device__ __forceinline__ uint32_t idesc_u8(uint32_t M, uint32_t N) {
    return (2u << 4) | ((N >> 3) << 17) | ((M >> 4) << 24);
}

__device__ __forceinline__ void mma_u8(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc,
                                       uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
        "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
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

// shared memory of one CTA handling up to maxc candidates per node
struct TcLayout {
    uint32_t rows, nodev, cid, cd, sid, sd, nrm, pby, bmask, chosen, bar, misc, bytes;
    __host__ __device__ static TcLayout make(uint32_t D, uint32_t maxc) {
        TcLayout l;
        l.rows   = 0;                  // maxc x D bytes, canonical layout, sorted order
        l.nodev  = l.rows + maxc * D;  // D bytes
        l.cid    = l.nodev + ((D + 15) & ~15u);
        l.cd     = l.cid + 4 * maxc;  // candidate order (A then B)
        l.sid    = l.cd + 4 * maxc;   // sorted order: id (top bit: a B candidate), distance,
        l.sd     = l.sid + 4 * maxc;  // squared norm
        l.nrm    = l.sd + 4 * maxc;
        l.pby    = l.nrm + 4 * maxc;  // [maxc / 32][maxc] bits of the candidates that prune t
        l.bmask  = l.pby + maxc * maxc / 8;  // sorted positions holding B candidates
        l.chosen = l.bmask + maxc / 8;       // the node's new list
        l.bar    = l.chosen + 4 * kMaxR;
        l.misc   = l.bar + 8;
        l.bytes  = l.misc + 4 * 16;
        return l;
    }
};

// Nodes are the slots in_list[0 .. *in_count) (or 0 .. n_nodes when in_list is
// null); nodes with more than MAXC candidates go to out_list.  COLS: TMEM columns per
// CTA, the width of a Gram tile.
template <uint32_t MAXC, uint32_t COLS>
__global__ void __launch_bounds__(kThreads, MAXC == 128 ? 8 : 1)
    prune_tc_kernel(PruneArgs a, uint32_t* counter, const uint32_t* in_list, const uint32_t* in_count,
                    uint32_t* out_list, uint32_t* out_count) {
    constexpr uint32_t KPT = MAXC / kThreads;  // candidates per thread
    constexpr uint32_t kB  = 0x80000000u;      // sid: a B candidate (ids are below 2^31)
    extern __shared__ __align__(1024) unsigned char smem[];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint64_t nwork = in_list ? (uint64_t)*reinterpret_cast<volatile const uint32_t*>(in_count) : a.n_nodes;
    if (nwork == 0) return;
    if (*reinterpret_cast<volatile const uint32_t*>(a.gate) != 0u) {  // rows not exact: hand every node on
        for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + tid; i < nwork; i += (uint64_t)gridDim.x * blockDim.x)
            out_list[atomicAdd(out_count, 1u)] = in_list ? __ldg(in_list + i) : (uint32_t)i;
        return;
    }

    const uint32_t D = a.D, R = a.R;
    const TcLayout lay = TcLayout::make(D, MAXC);
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
    uint32_t*      misc   = reinterpret_cast<uint32_t*>(smem + lay.misc);  // [0] tmem, [1] degree, [2..13] work items
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
    const uint32_t nchunk = D / 16;
    const uint32_t inv_nc = 0xFFFFFFFFu / nchunk + 1u;  // x / nchunk = __umulhi(x, inv_nc), nchunk >= 2
    const uint32_t LBO = 128, SBO = 8 * D;  // 8 rows x 16 B per core matrix; chunks adjacent
    const uint32_t ksteps = D / 32;         // kind::i8: K = 32 per instruction
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
        if (computed) {
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
            for (uint32_t c0 = 0; c0 < nc; c0 += 32) {             // the warp's own chunk: 128 q + 32 warp
                const uint4* dj = reinterpret_cast<const uint4*>(cd + c0);
                uint32_t     thr[KPT];
#pragma unroll
                for (uint32_t q = 0; q < KPT; ++q) thr[q] = b[q] + (c0 < 128u * q + 32u * warp ? 1u : 0u);
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
        for (uint32_t x = tid; x < m * nchunk; x += kThreads) {
            const uint32_t t = __umulhi(x, inv_nc), c = x - t * nchunk;
            cp_async16(rows_s + (t >> 3) * SBO + c * LBO + (t & 7u) * 16u,
                       a.vecs_u8 + (uint64_t)(sid[t] & ~kB) * D + 16u * c);
        }
        if (a.consistent) {
#pragma unroll
            for (uint32_t q = 0; q < KPT; ++q) {
                const uint32_t t    = 128u * q + tid;
                const uint32_t bits = __ballot_sync(0xffffffffu, t < m && (sid[t] & kB) != 0u);
                if (lane == 0) bmask[4u * q + warp] = bits;
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
            const uint32_t id   = idesc_u8(128u, N);
            for (uint32_t s = 0; s < ksteps; ++s) {
                const uint64_t da = umma_desc(rows_s + r * 16u * SBO + s * 2u * LBO, LBO, SBO);
                const uint64_t db = umma_desc(rows_s + c * (COLS / 8u) * SBO + s * 2u * LBO, LBO, SBO);
                mma_u8(tmem, da, db, id, s > 0 ? 1u : 0u);
            }
            mma_commit(bar);
        };
        if (m > 0 && tid == 0) {
            tc_fence_after();
            issue_tile(0, 0);
        }
        for (uint32_t t = tid; t < m; t += kThreads) {
            uint32_t n = 0;
            for (uint32_t c = 0; c < nchunk; ++c) {
                const uint4 v = *reinterpret_cast<const uint4*>(rows + (t >> 3) * SBO + c * LBO + (t & 7u) * 16u);
                n = dp4a_u(v.x, v.x, dp4a_u(v.y, v.y, dp4a_u(v.z, v.z, dp4a_u(v.w, v.w, n))));
            }
            nrm[t] = n;
        }
        __syncthreads();

        // --- 5. bits of the candidates that prune t
        bool late = false;
        for (uint32_t r = 0; r < nb; ++r) {
            const uint32_t t = 128u * r + tid;
            // "u prunes t" is alpha * d(u, t) <= d(node, t) in FP32, with d(u, t) the exact
            // integer Y = |u|^2 + |t|^2 - 2 u.t (< 2^24, so FP32 holds it exactly).  fl(Y *
            // alpha) does not decrease as Y grows, so the test is Y <= Ymax(t), the largest
            // integer with fl(Ymax * alpha) <= d(node, t): 2 u.t - |u|^2 >= |t|^2 - Ymax(t).
            int      thr  = 0;
            uint32_t keep = ~0u;  // consistent lists: no B candidate is checked against another
            if (t < m) {
                const float sdt = sd[t];
                int         y   = (int)fminf(floorf(sdt / a.alpha), 16777215.f);
                while (y < 16777215 && (float)(y + 1) * a.alpha <= sdt) ++y;
                while (y > 0 && (float)y * a.alpha > sdt) --y;
                thr = (int)nrm[t] - y;
                if (a.consistent && (sid[t] & kB)) keep = 0u;
            }
            const uint32_t last  = 128u * r + 32u * warp + 31u;  // the warp's last candidate
            const uint32_t ncols = min(m, 128u * (r + 1u));
            for (uint32_t c = 0; COLS * c < ncols; ++c) {
                if (r != 0 || c != 0) {
                    tc_fence_before();
                    __syncthreads();  // every thread's reads of the previous tile are done
                    if (tid == 0) {
                        tc_fence_after();
                        issue_tile(r, c);
                    }
                }
                late |= !mbar_wait(bar, phase);
                phase ^= 1u;
                tc_fence_after();
#pragma unroll 1
                for (uint32_t c32 = 0; c32 < COLS; c32 += 32u) {
                    const uint32_t u0 = COLS * c + c32;
                    if (u0 >= m || u0 > last) break;
                    uint32_t word = 0;
#pragma unroll
                    for (uint32_t h = 0; h < 32u; h += 16u) {
                        if (u0 + h < m) {
                            uint32_t g[16];
                            tmem_ld16(tmem + ((32u * warp) << 16) + c32 + h, g);
#pragma unroll
                            for (uint32_t k = 0; k < 16; k += 4) {
                                const uint4 nu = *reinterpret_cast<const uint4*>(nrm + u0 + h + k);
                                word |= (uint32_t)((int)(2u * g[k] - nu.x) >= thr) << (h + k);
                                word |= (uint32_t)((int)(2u * g[k + 1] - nu.y) >= thr) << (h + k + 1);
                                word |= (uint32_t)((int)(2u * g[k + 2] - nu.z) >= thr) << (h + k + 2);
                                word |= (uint32_t)((int)(2u * g[k + 3] - nu.w) >= thr) << (h + k + 3);
                            }
                        }
                    }
                    if (keep == 0u) word &= ~bmask[u0 >> 5];
                    if (t < m) pby[(u0 >> 5) * MAXC + t] = word;
                }
            }
        }
        tc_fence_before();
        if (__syncthreads_or(late)) {  // a wait for the tensor cores gave up
            failed = true;
            break;
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
    if (tid == 0 && a.pruned && done) atomicAdd(a.pruned, (unsigned long long)done);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS));
    }
}

}  // namespace

bool prune_tc_supported(uint32_t D, uint32_t R) { return D % 32 == 0 && D >= 32 && D <= 256 && R <= kMaxR; }

namespace {

template <uint32_t MAXC, uint32_t COLS>
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
    size_t       smem        = TcLayout::make(a.D, MAXC).bytes;
    const size_t floor_bytes = (size_t)(per_sm_smem / (max_ctas + 1) - reserved + 1024);
    if (smem < floor_bytes) smem = floor_bytes;
    auto kern = prune_tc_kernel<MAXC, COLS>;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
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
    kern<<<(unsigned)grid, kThreads, smem, st>>>(a, counter, in_list, in_count, out_list, out_count);
    return cudaGetLastError();
}

}  // namespace

// Passes of 128 candidates (up to 8 CTAs per SM), 256 (4), 512 (2), then 768 (one per
// SM, when its shared memory fits: D <= 160), each over the nodes the previous one
// handed on.  The first pass takes in_list[0 .. *in_count) (every node when null);
// what the last cannot take goes to out_list for prune_kernel.  A launch of no more
// nodes than SMs has nothing to fill with small passes: it goes straight to the last.
// ws: 2 * n_nodes + 4 words of device scratch; counters: four zeroed work counters.
cudaError_t launch_prune_tc(const PruneArgs& a, const uint32_t* in_list, const uint32_t* in_count,
                            uint32_t* out_list, uint32_t* out_count, uint32_t* ws, uint32_t* counters, int num_sms,
                            cudaStream_t st) {
    if (a.n_nodes == 0) return cudaSuccess;
    if (!prune_tc_supported(a.D, a.R) || !a.vecs_u8 || !a.gate || !out_list || !out_count)
        return cudaErrorInvalidValue;
    int dev = 0, max_optin = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    const bool last768 = TcLayout::make(a.D, 768).bytes <= (uint32_t)max_optin;
    if ((e = cudaMemsetAsync(out_count, 0, sizeof(uint32_t), st)) != cudaSuccess) return e;
    if (last768 && a.n_nodes <= (uint64_t)num_sms)
        return launch_tc<768, 128>(a, counters, in_list, in_count, out_list, out_count, a.n_nodes, num_sms, st);
    // the hand-off lists alternate between two halves of ws; their counts sit together
    uint32_t* list[2] = {ws, ws + a.n_nodes};
    uint32_t* cnt     = ws + 2 * a.n_nodes;  // one per hand-off
    if ((e = cudaMemsetAsync(cnt, 0, 3 * sizeof(uint32_t), st)) != cudaSuccess) return e;
    e = launch_tc<128, 64>(a, counters, in_list, in_count, list[0], cnt, a.n_nodes, num_sms, st);
    if (e != cudaSuccess) return e;
    e = launch_tc<256, 128>(a, counters + 1, list[0], cnt, list[1], cnt + 1, a.n_nodes, num_sms, st);
    if (e != cudaSuccess) return e;
    if (!last768) return launch_tc<512, 128>(a, counters + 2, list[1], cnt + 1, out_list, out_count, a.n_nodes, num_sms, st);
    e = launch_tc<512, 128>(a, counters + 2, list[1], cnt + 1, list[0], cnt + 2, a.n_nodes, num_sms, st);
    if (e != cudaSuccess) return e;
    return launch_tc<768, 128>(a, counters + 3, list[0], cnt + 2, out_list, out_count, a.n_nodes, num_sms, st);
}

}  // namespace vann
