// prune_rev.cu -- the reverse-edge re-prune for alpha-consistent lists, one warp
// per node.
//
// After a batch, each node v that received reverse entries is re-pruned over
// A = its new reverse sources and B = its current out-neighbours
// (pruneReverseEdges, vamana/include/kernels.cuh:626-743; candidate order and the
// rule as in prune.cu).  When B came out of RobustPrune with the same alpha, no
// B candidate prunes another, so the selection only needs the distances that
// involve an A candidate: |A| x |C| of them, not |C|^2.
//
//   1. a pass of gathers gives d(v, c) and d(a, c) of the first A candidate for every
//      candidate c, further passes two A candidates each (a pass per query loaded every row
//      twice; 11 re-prune passes of a 100k x 96 float build 3.83 -> 3.09 ms);
//   2. the candidates are ordered by (distance, index): B is already in that order
//      (it is a RobustPrune selection), so the A candidates are merged in by rank;
//   3. bit masks over the sorted positions: PA[i] = what A_i prunes,
//      SB[i] = the B candidates that prune A_i;
//   4. selection, all on those masks: every live B candidate ahead of the next
//      live A candidate is chosen in one step; that A candidate is chosen unless
//      a chosen B candidate prunes it, and then removes what it prunes.
// This gives the same list as evaluating every pair (prune.cu).  Distances use the
// exact uint8 rows when they are exact (dp4a), else the FP32 rows, in the same
// summation order as prune_kernel.  Nodes with more than kMaxC candidates or
// kMaxA reverse sources are handed on in out_list.
#include "common.cuh"
#include "kernels.h"

namespace vann {
namespace {

constexpr uint32_t kMaxC = 128;  // candidates per node
constexpr uint32_t kMaxA = 8;    // reverse sources per node
constexpr uint32_t kW    = kMaxC / 32;

struct RevWarp {  // shared memory of one warp
    uint32_t cid[kMaxC];
    uint32_t hash[kMaxC];       // their filter slots
    float    cd[kMaxC];
    uint64_t keys[kMaxC];
    float    ad[kMaxA][kMaxC];  // d(A_i, candidate j)
    uint32_t pa[kMaxA][kW];     // sorted positions A_i prunes
    uint32_t sb[kMaxA][kW];     // sorted positions of B candidates that prune A_i
};

// the query `qid` in the row format the distances use (uint8 rows: the exact uint8 row itself)
template <typename S, int DC>
__device__ __forceinline__ void load_node(Query<S, DC>& q, const PruneArgs& a, uint32_t qid, uint32_t lane) {
    if constexpr (S::kInt) load_query_u8row<S, DC>(q, a.vecs_u8 + (uint64_t)qid * a.D, a.D, lane);
    else load_query<S, DC>(q, a.vecs + (uint64_t)qid * a.D, a.D, lane);
}

// Squared distances of two queries to the same round of rows, as dist_round gives them one
// by one (the sums are taken in its order): the rows are loaded once, and a uint8 row's
// own norm is formed once.
template <typename S, int DC>
__device__ __forceinline__ void dist_round2(const Query<S, DC>& q0, const Query<S, DC>& q1, const void* base,
                                            const uint32_t* ids, int cnt, uint32_t D, uint32_t lane, float* out0,
                                            float* out1) {
    using Ly                 = Layout<S, DC>;
    constexpr int  M         = Ly::kM;
    const uint32_t chunks    = D / S::kElems;
    const uint64_t row_bytes = (uint64_t)D * 16u / (uint64_t)S::kElems;
    const uint32_t t = lane % Ly::kT, g = lane / Ly::kT;
    uint4          x[M][Ly::kCPL];
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const int      r     = m * Ly::kP + (int)g;
        const bool     valid = r < cnt;
        const uint32_t id    = valid ? ids[r] : 0u;
#pragma unroll
        for (int c = 0; c < Ly::kCPL; ++c) x[m][c] = make_uint4(0u, 0u, 0u, 0u);
        if (m * Ly::kP >= cnt) continue;
        if constexpr (Ly::kNarrow) {
            const uint32_t k0 = Ly::chunk(t, 0);
            if (valid && k0 + 1u < chunks && (row_bytes & 31u) == 0u) {
                load32(base, row_bytes, id, k0, x[m][0], x[m][1]);
            } else {
                if (valid && k0 < chunks) x[m][0] = load16(base, row_bytes, id, k0);
                if (valid && k0 + 1u < chunks) x[m][1] = load16(base, row_bytes, id, k0 + 1u);
            }
        } else {
#pragma unroll
            for (int c = 0; c < Ly::kCPL; ++c) {
                const uint32_t k = Ly::chunk(t, c);
                if (valid && k < chunks) x[m][c] = load16(base, row_bytes, id, k);
            }
        }
    }
    float y0, y1;
    if constexpr (S::kInt) {
        int v0[M], v1[M];
#pragma unroll
        for (int m = 0; m < M; ++m) {
            v0[m] = v1[m] = 0;
            if (m * Ly::kP >= cnt) continue;
            unsigned xx = 0u, a0 = 0u, a1 = 0u;
#pragma unroll
            for (int c = 0; c < Ly::kCPL; ++c) {
                const unsigned w[4] = {x[m][c].x, x[m][c].y, x[m][c].z, x[m][c].w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    xx = __dp4a(w[i], w[i], xx);
                    a0 = __dp4a((unsigned)q0.u[c][i], w[i], a0);
                    a1 = __dp4a((unsigned)q1.u[c][i], w[i], a1);
                }
            }
            v0[m] = (int)xx - 2 * (int)a0;
            v1[m] = (int)xx - 2 * (int)a1;
        }
        y0 = (float)(group_reduce<M, Ly::kT, int>(v0, lane) + q0.qq);
        y1 = (float)(group_reduce<M, Ly::kT, int>(v1, lane) + q1.qq);
    } else {
        const float2 neg1 = make_float2(-1.f, -1.f);
        float2       s0[M], s1[M];
#pragma unroll
        for (int m = 0; m < M; ++m) s0[m] = s1[m] = make_float2(0.f, 0.f);
#pragma unroll
        for (int c = 0; c < Ly::kCPL; ++c) {
#pragma unroll
            for (int m = 0; m < M; ++m) {
                float2 e[S::kElems / 2];
                S::widen2(x[m][c], e);
#pragma unroll
                for (int p = 0; p < S::kElems / 2; ++p) {
                    float2 d = __ffma2_rn(q0.f2[c][p], neg1, e[p]);
                    s0[m]    = __ffma2_rn(d, d, s0[m]);
                    d        = __ffma2_rn(q1.f2[c][p], neg1, e[p]);
                    s1[m]    = __ffma2_rn(d, d, s1[m]);
                }
            }
        }
        float v0[M], v1[M];
#pragma unroll
        for (int m = 0; m < M; ++m) {
            v0[m] = s0[m].x + s0[m].y;
            v1[m] = s1[m].x + s1[m].y;
        }
        y0 = group_reduce<M, Ly::kT, float>(v0, lane);
        y1 = group_reduce<M, Ly::kT, float>(v1, lane);
    }
    const uint32_t vi = round_row_of_lane<S, DC>(lane);
    if (round_writer<S, DC>(lane) && (int)vi < cnt) {
        out0[vi] = y0;
        out1[vi] = y1;
    }
}

// distances of every candidate to the node and to every A candidate, two of these queries
// to a pass over the candidates' rows (most nodes have one A candidate: one pass)
template <typename S, int DC>
__device__ __forceinline__ void all_dists(const PruneArgs& a, const void* store, RevWarp& w, uint32_t node,
                                          uint32_t nA, uint32_t nc, uint32_t lane) {
    constexpr uint32_t G = Layout<S, DC>::kG;
    for (uint32_t i = 0; i <= nA; i += 2) {  // query 0 is the node, query i + 1 is A_i
        Query<S, DC> q0, q1;
        load_node<S, DC>(q0, a, i == 0u ? node : w.cid[i - 1u], lane);
        float* out0 = i == 0u ? w.cd : w.ad[i - 1u];
        if (i < nA) {
            load_node<S, DC>(q1, a, w.cid[i], lane);
            for (uint32_t g0 = 0; g0 < nc; g0 += G)
                dist_round2<S, DC>(q0, q1, store, w.cid + g0, (int)min(G, nc - g0), a.D, lane, out0 + g0, w.ad[i] + g0);
        } else {
            // uint8 rows are used only when every row is exact, so the query row is integer-valued
            for (uint32_t g0 = 0; g0 < nc; g0 += G)
                dist_round<S, DC, S::kInt>(q0, store, nullptr, [&](int j) { return w.cid[g0 + j]; },
                                           (int)min(G, nc - g0), a.D, lane, out0 + g0);
        }
    }
}

// U8: distances from the exact uint8 rows (chosen on the host, which has read the
// exactness flag); the kernel then holds one distance path only, which keeps its code
// small enough for the instruction cache.  Should the flag say otherwise on the device,
// every node is handed on to the next pass.
template <int DC, bool U8>
__global__ void __launch_bounds__(128) prune_rev_kernel(PruneArgs a, uint32_t* out_list, uint32_t* out_count) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const uint32_t lane = threadIdx.x & 31u;
    RevWarp&       w    = reinterpret_cast<RevWarp*>(smem_raw)[threadIdx.x >> 5];
    const uint32_t R    = a.R;
    const bool     gated = U8 && (a.vecs_u8 == nullptr || a.gate == nullptr ||
                                  *reinterpret_cast<volatile const uint32_t*>(a.gate) != 0u);
    uint32_t       done = 0;

    for (;;) {
        uint32_t s = 0;
        if (lane == 0) s = atomicAdd(a.counter, 1u);
        s = __shfl_sync(0xffffffffu, s, 0);
        if (s >= a.n_nodes) break;
        const uint32_t node = __ldg(a.node_ids + s);
        if (node == kNone) continue;  // the padded slots' run in the sorted edge list
        const uint32_t ci   = a.csr_by_slot ? s : node;
        const uint32_t nA   = min(__ldg(a.csr_cnt + ci), a.cap);
        const uint32_t aoff = __ldg(a.csr_off + ci);
        const uint32_t nB   = a.use_b ? min(a.deg[node], R) : 0u;
        const uint32_t nc   = nA + nB;
        if (nc > kMaxC || nA > kMaxA || gated) {
            if (lane == 0) out_list[atomicAdd(out_count, 1u)] = s;
            continue;
        }
        for (uint32_t i = lane; i < nc; i += 32) {
            const uint64_t e = (uint64_t)node * R + (i - nA);
            w.cid[i]         = i < nA ? __ldg(a.csr_src + aoff + i) : a.adj[e];
            if (i >= nA) w.hash[i] = a.adj_h[e];
        }
        __syncwarp();

        // --- 1. distances
        if constexpr (U8) all_dists<StoreU8, DC>(a, a.vecs_u8, w, node, nA, nc, lane);
        else all_dists<StoreF32, DC>(a, a.vecs, w, node, nA, nc, lane);
        __syncwarp();

        // --- 2. stable order by (distance, candidate index)
        uint32_t p2 = 32;
        while (p2 < nc) p2 <<= 1;
        // B came out of RobustPrune in selection order: nondecreasing distance, ties in
        // list order, which is also their index order here.  Then the order is B with
        // the A candidates merged in (every A index is below every B index):
        //   B_j goes to j + #{i : d(A_i) <= d(B_j)},
        //   A_i to #{j : d(B_j) < d(A_i)} + #{k : (d(A_k), k) < (d(A_i), i)}.
        // A list out of order (a graph set from outside) takes the bitonic sort.
        // Distances compare by their bits, the keys' order (non-negative; a NaN sorts last: as
        // floats it would leave a position unwritten).
        auto dist_bits = [&](uint32_t j) { return __float_as_uint(w.cd[j]); };
        bool in_order  = true;
        for (uint32_t j = lane; j + 1u < nB; j += 32) in_order &= dist_bits(nA + j) <= dist_bits(nA + j + 1u);
        if (__all_sync(0xffffffffu, in_order)) {
            for (uint32_t j = lane; j < nB; j += 32) {
                const uint32_t d   = dist_bits(nA + j);
                uint32_t       pos = j;
                for (uint32_t i = 0; i < nA; ++i) pos += dist_bits(i) <= d ? 1u : 0u;
                w.keys[pos] = make_key(w.cd[nA + j], nA + j);
            }
            for (uint32_t i = 0; i < nA; ++i) {
                const uint32_t di  = dist_bits(i);
                uint32_t       pos = 0;
                for (uint32_t j0 = 0; j0 < nB; j0 += 32) {
                    const uint32_t j = j0 + lane;
                    pos += __popc(__ballot_sync(0xffffffffu, j < nB && dist_bits(nA + j) < di));
                }
                for (uint32_t k = 0; k < nA; ++k) {
                    const uint32_t dk = dist_bits(k);
                    pos += (dk < di || (dk == di && k < i)) ? 1u : 0u;
                }
                if (lane == 0) w.keys[pos] = make_key(w.cd[i], i);
            }
            for (uint32_t i = nc + lane; i < p2; i += 32) w.keys[i] = ~0ull;
            __syncwarp();
        } else {
            for (uint32_t i = lane; i < p2; i += 32) w.keys[i] = i < nc ? make_key(w.cd[i], i) : ~0ull;
            __syncwarp();
            warp_bitonic_sort_smem(w.keys, p2, lane);
        }
        const uint32_t m = min(nc, a.cap);

        // --- 3. masks over sorted positions t < m (position t = 32k + lane)
        uint32_t am[kW];  // positions holding A candidates
#pragma unroll
        for (uint32_t k = 0; k < kW; ++k) {
            const uint32_t t   = 32u * k + lane;
            const uint32_t idx = t < m ? (uint32_t)w.keys[t] : 0u;
            am[k]              = __ballot_sync(0xffffffffu, t < m && idx < nA);
        }
        for (uint32_t i = 0; i < nA; ++i) {
            const float di = w.cd[i];
#pragma unroll
            for (uint32_t k = 0; k < kW; ++k) {
                const uint32_t t   = 32u * k + lane;
                bool           pr = false, by = false;
                if (t < m) {
                    const uint32_t idx = (uint32_t)w.keys[t];
                    const float    y   = w.ad[i][idx] * a.alpha;
                    pr                 = y <= w.cd[idx];           // A_i prunes the candidate at t
                    by                 = idx >= nA && y <= di;     // the B candidate at t prunes A_i
                }
                const uint32_t bp = __ballot_sync(0xffffffffu, pr), bb = __ballot_sync(0xffffffffu, by);
                if (lane == 0) {
                    w.pa[i][k] = bp;
                    w.sb[i][k] = bb;
                }
            }
        }
        __syncwarp();

        // --- 4. selection (the same on every lane).  Candidates are chosen in sorted order,
        // so the new list is the chosen positions in ascending order, the first R.
        uint32_t live[kW], sel[kW], chosen_b[kW];
#pragma unroll
        for (uint32_t k = 0; k < kW; ++k) {
            const uint32_t lo = 32u * k;
            live[k]           = m >= lo + 32u ? ~0u : (m > lo ? (1u << (m - lo)) - 1u : 0u);
            sel[k] = chosen_b[k] = 0u;
        }
        uint32_t ndeg = 0;
        for (;;) {
            uint32_t tA = m;  // next live A candidate
#pragma unroll
            for (int k = kW - 1; k >= 0; --k)
                if (live[k] & am[k]) tA = 32u * (uint32_t)k + __ffs(live[k] & am[k]) - 1u;
            // live B candidates ahead of it: all chosen, in order
#pragma unroll
            for (uint32_t k = 0; k < kW; ++k) {
                const uint32_t lo   = 32u * k;
                const uint32_t mask = tA >= lo + 32u ? ~0u : (tA > lo ? (1u << (tA - lo)) - 1u : 0u);
                const uint32_t run  = live[k] & ~am[k] & mask;
                sel[k] |= run;
                chosen_b[k] |= run;
                live[k] &= ~run;
                ndeg += __popc(run);
            }
            if (ndeg >= R || tA >= m) break;
            // decide the A candidate at tA
            const uint32_t i = (uint32_t)w.keys[tA];
            bool           pruned = false;
#pragma unroll
            for (uint32_t k = 0; k < kW; ++k) pruned |= (w.sb[i][k] & chosen_b[k]) != 0u;
#pragma unroll
            for (uint32_t k = 0; k < kW; ++k) {
                const uint32_t bit = k == (tA >> 5) ? 1u << (tA & 31u) : 0u;
                live[k] &= ~bit;
                if (!pruned) {
                    sel[k] |= bit;
                    live[k] &= ~w.pa[i][k];
                }
            }
            if (!pruned && ++ndeg >= R) break;
        }
        ndeg = min(ndeg, R);
        // the list; a slot that keeps its entry is not written.  Filter slots come from the
        // node's row, only an A candidate's are computed (two 64-bit remainders: computed
        // for every entry at each step above they took a fifth of the kernel: 30 re-prune
        // passes of a 300k x 128 uint8 build 16.0 -> 12.6 ms)
        {
            const uint64_t out  = (uint64_t)node * R;
            uint32_t       rank = 0;
#pragma unroll
            for (uint32_t k = 0; k < kW; ++k) {
                const uint32_t r = rank + __popc(sel[k] & ((1u << lane) - 1u));
                if (((sel[k] >> lane) & 1u) && r < R) {
                    const uint32_t i  = (uint32_t)w.keys[32u * k + lane];
                    const uint32_t id = w.cid[i];
                    if (r >= nB || w.cid[nA + r] != id) {
                        a.adj[out + r]   = id;
                        a.adj_h[out + r] = i < nA ? bloom_pack(id) : w.hash[i];
                    }
                }
                rank += __popc(sel[k]);
            }
        }
        if (lane == 0) a.deg[node] = ndeg;
        ++done;
        __syncwarp();
    }
    if (lane == 0 && a.pruned && done) atomicAdd(a.pruned + 1, (unsigned long long)done);
}

}  // namespace

cudaError_t launch_prune_rev(const PruneArgs& a, bool u8, uint32_t* out_list, uint32_t* out_count, int num_sms,
                             cudaStream_t st) {
    if (a.n_nodes == 0) return cudaSuccess;
    if (!a.node_ids || !a.csr_off || !a.consistent || a.D > 256) return cudaErrorInvalidValue;
    const int    warps = 4;
    const size_t smem  = sizeof(RevWarp) * warps;
    auto         kern  = a.D <= 128 ? (u8 ? prune_rev_kernel<0, true> : prune_rev_kernel<0, false>)
                                    : (u8 ? prune_rev_kernel<1, true> : prune_rev_kernel<1, false>);
    cudaError_t  e     = allow_smem(kern, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e          = fit_carveout(kern, warps * 32, smem, &per_sm);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    uint64_t grid = (uint64_t)per_sm * num_sms;
    const uint64_t need = (a.n_nodes + warps - 1) / warps;
    if (grid > need) grid = need;
    kern<<<(unsigned)grid, warps * 32, smem, st>>>(a, out_list, out_count);
    return cudaGetLastError();
}

}  // namespace vann
