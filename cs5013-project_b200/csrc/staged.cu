// staged.cu -- searchPoints2's merge of graph results with the insert list.
//
// Restates merge_and_rerank_kernel (vamana/include/utils.cuh:199-285) with the
// same decisions.  For each query the L graph worklist entries, then every staged
// (insert-list) row, compete for L slots in that order.  A candidate enters when its
// squared distance is strictly below the largest slot value, replacing the first
// slot that holds it.  The slots start at +inf and are finally put in stable
// distance order (the reference's bubble sort).
//
// The reference runs this on one thread per query.  Here a warp serves a query, several
// queries to a CTA:
//   * each lane computes one candidate's distance, sequentially over the dimensions
//     with one fused multiply-add each, as l2_distance_sq (:150-158) compiles;
//   * the L worklist entries fill the slots in order, since every slot starts at +inf;
//   * the insert-list rows pass through shared memory in tiles of 32 that all queries of
//     the CTA read, the next tile on its way meanwhile;
//   * a ballot of the 32 candidates against the current largest slot value selects
//     the few that can enter; they are applied in arrival order;
//   * the slot values are in registers (slot k: register k / 32 of lane k % 32), so a
//     replacement is the owning lane's rescan of its few and two warp reductions;
//   * the output order comes from counted ranks, and eight rows are copied out at a time.
// 1,000 queries, 500 list rows, L = 100, D = 128, rows returned: 113 us, where a lane reading
// its own list row from global memory, slots in shared memory (a replacement, 90 per query,
// was 900 cycles), a bitonic sort and one row copied at a time took 272.
#include "common.cuh"
#include "kernels.h"

namespace vann {
namespace {

constexpr uint32_t kStaged = 0x80000000u;

__device__ __forceinline__ float l2_seq(const float* q, const float* row, uint32_t D) {
    float d = 0.f;
#pragma unroll 8
    for (uint32_t i = 0; i < D; i += 4) {
        const float4 x = __ldg(reinterpret_cast<const float4*>(row + i));
        float        e = q[i] - x.x;
        d              = fmaf(e, e, d);
        e              = q[i + 1] - x.y;
        d              = fmaf(e, e, d);
        e              = q[i + 2] - x.z;
        d              = fmaf(e, e, d);
        e              = q[i + 3] - x.w;
        d              = fmaf(e, e, d);
    }
    return d;
}

// the same with the row in shared memory
__device__ __forceinline__ float l2_seq_shared(const float* q, const float* row, uint32_t D) {
    float d = 0.f;
#pragma unroll 4
    for (uint32_t i = 0; i < D; i += 4) {
        const float4 x = *reinterpret_cast<const float4*>(row + i);
        const float4 y = *reinterpret_cast<const float4*>(q + i);
        float        e = y.x - x.x;
        d              = fmaf(e, e, d);
        e              = y.y - x.y;
        d              = fmaf(e, e, d);
        e              = y.z - x.z;
        d              = fmaf(e, e, d);
        e              = y.w - x.w;
        d              = fmaf(e, e, d);
    }
    return d;
}

// (largest value, first slot holding it) over the warp; v = lane's largest (slot values are
// non-negative; -1 for a lane without slots, so their bits order them as integers), s = its
// first slot
__device__ __forceinline__ void warp_argmax(float& v, uint32_t& s) {
    const int b = __float_as_int(v);
    const int m = __reduce_max_sync(0xffffffffu, b);
    s           = __reduce_min_sync(0xffffffffu, b == m ? s : kNone);
    v           = __int_as_float(m);
}

constexpr uint32_t kTile     = 32;  // insert-list rows per tile, one per lane
constexpr uint32_t kMaxWarps = 8;

// J: slots per lane (L <= 32 J); slot k is register k / 32 of lane k % 32.
template <int J>
__global__ void __launch_bounds__(32 * kMaxWarps) staged_merge_kernel(StagedArgs a, uint32_t warp_bytes) {
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t wib  = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const uint32_t L = a.L, D = a.D;
    const uint32_t stride = D + 4u;  // floats: rows of a tile fall on different banks
    float*         tile   = reinterpret_cast<float*>(smem);  // two tiles
    unsigned char* base   = smem + 8u * kTile * stride + (size_t)wib * warp_bytes;
    float*         qv     = reinterpret_cast<float*>(base);           // D
    float*         sd     = qv + D;                                     // slot values
    uint32_t*      sid    = reinterpret_cast<uint32_t*>(sd + 32 * J);   // slot ids
    uint32_t*      perm   = reinterpret_cast<uint32_t*>(sid + 32 * J);  // slots in output order
    const uint32_t tiles  = (uint32_t)((a.n_stage + kTile - 1u) / kTile);
    const uint32_t chunks = D / 4u;

    auto load_tile = [&](uint32_t t) {  // rows 32 t .. into buffer t & 1
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(tile + (t & 1u) * kTile * stride);
        for (uint32_t r = wib; r < kTile; r += warps) {
            const uint64_t row = (uint64_t)t * kTile + r;
            if (row < a.n_stage)
                for (uint32_t c = lane; c < chunks; c += 32u)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 4u * (r * stride + 4u * c)),
                                 "l"(a.stage + row * D + 4u * c)
                                 : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    for (uint64_t q0 = blockIdx.x * (uint64_t)warps; q0 < a.nq; q0 += (uint64_t)gridDim.x * warps) {
        const uint64_t qi = q0 + wib;
        const bool     on = qi < a.nq;  // every warp takes part in loading the tiles
        if (tiles > 0u) load_tile(0);
        float    sv[J], lmax = -1.f, gmax = -1.f;
        uint32_t lslot = kNone, gslot = kNone;
        auto     lane_max = [&]() {  // this lane's largest slot value, first slot
            lmax  = -1.f;
            lslot = kNone;
#pragma unroll
            for (int j = 0; j < J; ++j)
                if (sv[j] > lmax) {
                    lmax  = sv[j];
                    lslot = 32u * (uint32_t)j + lane;
                }
        };
        if (on) {
            for (uint32_t i = lane; i < D; i += 32) qv[i] = a.queries[qi * D + i];
            __syncwarp();
            // the worklist entries, in order, into the slots, all +inf at first
            uint32_t n = 0;
            for (uint32_t c0 = 0; c0 < L; c0 += 32) {
                const uint32_t c  = c0 + lane;
                const uint32_t id = c < L ? a.graph_ids[qi * L + c] : kNone;
                float          d  = __int_as_float(0x7f800000);
                if (id != kNone) d = l2_seq(qv, a.vecs + (uint64_t)id * D, D);
                const bool     in = d < __int_as_float(0x7f800000);
                const uint32_t m  = __ballot_sync(0xffffffffu, in);
                const uint32_t k  = n + __popc(m & ((1u << lane) - 1u));
                if (in) {
                    sd[k]  = d;
                    sid[k] = id;
                }
                n += __popc(m);
            }
            for (uint32_t k = n + lane; k < L; k += 32) {
                sd[k]  = __int_as_float(0x7f800000);
                sid[k] = kNone;
            }
            __syncwarp();
#pragma unroll
            for (int j = 0; j < J; ++j) sv[j] = 32u * (uint32_t)j + lane < L ? sd[32u * (uint32_t)j + lane] : -1.f;
            lane_max();
            gmax  = lmax;
            gslot = lslot;
            warp_argmax(gmax, gslot);
        }

        for (uint32_t t = 0; t < tiles; ++t) {
            if (t + 1u < tiles) {
                load_tile(t + 1u);
                asm volatile("cp.async.wait_group 1;" ::: "memory");
            } else {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
            __syncthreads();
            if (on) {
                const uint64_t s   = (uint64_t)t * kTile + lane;
                const float*   row = tile + ((t & 1u) * kTile + lane) * stride;
                const uint32_t id  = kStaged | (uint32_t)s;
                float          d   = __int_as_float(0x7f800000);
                if (s < a.n_stage) d = l2_seq_shared(qv, row, D);
                uint32_t m = __ballot_sync(0xffffffffu, d < gmax);
                while (m) {
                    const uint32_t src = __ffs(m) - 1u;
                    m &= m - 1u;
                    const float dc = __shfl_sync(0xffffffffu, d, src);
                    if (!(dc < gmax)) continue;  // the largest value dropped meanwhile
                    const uint32_t idc = __shfl_sync(0xffffffffu, id, src);
                    if (lane == (gslot & 31u)) {
                        sid[gslot] = idc;
#pragma unroll
                        for (int j = 0; j < J; ++j)
                            if (gslot == 32u * (uint32_t)j + lane) sv[j] = dc;
                        lane_max();
                    }
                    gmax  = lmax;
                    gslot = lslot;
                    warp_argmax(gmax, gslot);
                }
            }
            __syncthreads();  // the buffer is free
        }
        if (!on) continue;  // no barrier after this in the round
        __syncwarp();
        // stable order by distance (+inf slots last): each slot's rank by counting
#pragma unroll
        for (int j = 0; j < J; ++j)
            if (32u * (uint32_t)j + lane < L) sd[32u * (uint32_t)j + lane] = sv[j];
        __syncwarp();
        uint32_t rank[J];
#pragma unroll
        for (int j = 0; j < J; ++j) rank[j] = 0u;
        for (uint32_t k = 0; k < L; ++k) {
            const float d = sd[k];
#pragma unroll
            for (int j = 0; j < J; ++j)
                rank[j] += (d < sv[j] || (d == sv[j] && k < 32u * (uint32_t)j + lane)) ? 1u : 0u;
        }
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const uint32_t k = 32u * (uint32_t)j + lane;
            if (k < L) {
                a.out_ids[qi * L + rank[j]] = sid[k];
                a.out_d[qi * L + rank[j]]   = sv[j];
                perm[rank[j]]               = k;
            }
        }
        __syncwarp();
        if (a.out_vecs) {
            auto row_of = [&](uint32_t t) -> const float* {
                const uint32_t id = sid[perm[t]];
                return id == kNone ? nullptr
                     : (id & kStaged) ? a.stage + (uint64_t)(id & ~kStaged) * D
                                      : a.vecs + (uint64_t)id * D;
            };
            if ((reinterpret_cast<uintptr_t>(a.out_vecs) & 15u) == 0u) {
                // eight rows on their way at a time
                for (uint32_t t0 = 0; t0 < L; t0 += 8u) {
                    const float* src[8];
#pragma unroll
                    for (uint32_t r = 0; r < 8; ++r) src[r] = t0 + r < L ? row_of(t0 + r) : nullptr;
                    for (uint32_t i = 4u * lane; i < D; i += 128u) {
                        float4 x[8];
#pragma unroll
                        for (uint32_t r = 0; r < 8; ++r)
                            x[r] = src[r] ? __ldg(reinterpret_cast<const float4*>(src[r] + i))
                                          : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                        for (uint32_t r = 0; r < 8; ++r)
                            if (t0 + r < L)
                                *reinterpret_cast<float4*>(a.out_vecs + (qi * L + t0 + r) * D + i) = x[r];
                    }
                }
            } else {
                for (uint32_t t = 0; t < L; ++t) {
                    const float* src = row_of(t);
                    for (uint32_t i = lane; i < D; i += 32)
                        a.out_vecs[(qi * L + t) * D + i] = src ? __ldg(src + i) : 0.f;
                }
            }
        }
        __syncwarp();
    }
}

template <int J>
cudaError_t launch_staged_j(const StagedArgs& a, int num_sms, cudaStream_t st) {
    int         dev = 0, optin = 0;
    cudaError_t e   = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    const uint32_t warp_bytes = (4u * a.D + 3u * 4u * 32u * J + 15u) & ~15u;
    const size_t   tile_bytes = 8ull * kTile * (a.D + 4u);
    // queries per CTA: as many as share a tile well, but enough CTAs for every SM
    int warps = (int)kMaxWarps;
    while (warps > 1 && (tile_bytes + (size_t)warps * warp_bytes > (size_t)optin ||
                         (a.nq + warps - 1) / warps < (uint64_t)num_sms))
        warps >>= 1;
    const size_t smem = tile_bytes + (size_t)warps * warp_bytes;
    auto         kern = staged_merge_kernel<J>;
    e                 = allow_smem(kern, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e          = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, warps * 32, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    uint64_t       grid = (uint64_t)per_sm * num_sms;
    const uint64_t need = (a.nq + warps - 1) / warps;
    if (grid > need) grid = need;
    kern<<<(unsigned)grid, warps * 32, smem, st>>>(a, warp_bytes);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_staged_merge(const StagedArgs& a, int num_sms, cudaStream_t st) {
    if (a.nq == 0 || a.L == 0) return cudaSuccess;
    if (a.L <= 128) return launch_staged_j<4>(a, num_sms, st);
    if (a.L <= 256) return launch_staged_j<8>(a, num_sms, st);
    if (a.L <= 1024) return launch_staged_j<32>(a, num_sms, st);
    return cudaErrorInvalidValue;
}

}  // namespace vann
