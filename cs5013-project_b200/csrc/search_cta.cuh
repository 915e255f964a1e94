// search_cta.cuh -- GreedySearch with one CTA of 5 warps per query, for batches that
// leave the chip mostly idle.
//
// Same semantics and results as search_kernel (search_impl.cuh), restating the
// reference's GreedySearch (vamana/include/search.cuh:20-367).  A query is a chain of
// dependent hops, and with few queries the length of that chain is the time: one warp
// takes a hop's list, filter, row gathers, merge and next parent one after the other.
// Here the chain holds only what the next hop waits for:
//   * warps 1-4 gather a quarter of the new rows each (FP32 rows in one round instead of
//     four);
//   * the next parent is the best candidate that can enter the worklist or the first
//     unvisited entry, whichever is closer, which needs the new distances and two values
//     of the worklist but not their merge.  Warps 1 .. SPL each take it for themselves and
//     filter 32 slots of its list;
//   * warp 0 owns the worklist (in registers, L <= 256) and merges hop h's candidates
//     while the others are on hop h + 1; it also requests the lists of the candidates it
//     keeps, the parents to come, into L2.
// Per hop two barriers: one when the distances are there (and the previous merge is
// done), one of the gathering warps when the filtered list is there.  What passes between
// the two sides is double-buffered by hop parity.
#pragma once
#include "search_impl.cuh"

namespace vann {

constexpr uint32_t kCtaThreads = 160;  // warp 0: worklist; warps 1-4: gathers
constexpr uint32_t kCtaGather  = 4;

struct CtaSearchLayout {
    uint32_t lp;     // L rounded up to 32
    uint32_t slots;  // candidate slots of a hop
    uint32_t wl_id, wl_d, nb, srt, keys, ctl, bytes;  // ctl 16-byte aligned
    __host__ __device__ static CtaSearchLayout make(uint32_t L, uint32_t slots, bool rerank) {
        CtaSearchLayout s;
        s.lp    = (L + 31u) & ~31u;
        s.slots = slots;
        s.wl_id = 5008u;
        s.wl_d  = s.wl_id + 4u * s.lp;
        s.nb    = s.wl_d + 4u * s.lp;   // two buffers of candidate ids, then distances
        s.srt   = s.nb + 16u * slots;   // the merge's keys
        s.keys  = s.srt + 8u * slots;   // the rerank's keys
        s.ctl   = s.keys + (rerank ? 8u * s.lp : 0u);
        s.bytes = s.ctl + 4u * 20u;
        return s;
    }
};

// Rows per lane in a gather round here: a hop measures some 6 to 30 rows, a quarter of
// them per warp, so rounds of 4 (FP32) to 8 rows, where the warp-per-query kernels take 8
// to 32; fewer registers, more CTAs per SM, no arithmetic for rows that are not there.
template <typename S, int DC>
struct CtaRows {
    static constexpr int kWant = S::kInt ? 8 : 4;  // rows per round
    static constexpr int kP    = Layout<S, DC>::kP;
    static constexpr int kFit  = kWant >= kP ? kWant / kP : 1;
    static constexpr int kM    = kFit < Layout<S, DC>::kM ? kFit : Layout<S, DC>::kM;
};

// warps 1-4
__device__ __forceinline__ void gather_barrier() {
    asm volatile("bar.sync 1, %0;" ::"n"(32 * kCtaGather) : "memory");
}
// all warps, from the worklist's side and the gathering side: not __syncthreads, which every
// thread must reach at the same place
__device__ __forceinline__ void hop_barrier() { asm volatile("bar.sync 2, %0;" ::"n"(kCtaThreads) : "memory"); }
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// IQ: as in search_kernel.  strict: candidates enter only when strictly closer than the
// last entry, +inf while the list is not full (the register-worklist kernel's rule).
// LREG: worklist entries per lane of warp 0 (L <= 32 LREG).
template <typename S, int DC, int SPL, int LREG, bool IQ>
__global__ void __launch_bounds__(kCtaThreads, LREG <= 4 ? 4 : 3) search_cta_kernel(SearchArgs a, bool strict) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int         M     = CtaRows<S, DC>::kM;
    constexpr uint32_t    G     = M * Layout<S, DC>::kP;
    constexpr uint32_t    SLOTS = SPL * 32;
    constexpr uint32_t    kDone = 0xFFFFFFFFu;
    const float           kInf  = __int_as_float(0x7f800000);
    const uint32_t        open  = strict ? __float_as_uint(kInf) : kNone;  // tail of a list with room
    const uint32_t        tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const CtaSearchLayout lay   = CtaSearchLayout::make(a.L, SLOTS, a.rerank != 0);
    uint32_t*             bloom = reinterpret_cast<uint32_t*>(smem);
    uint32_t*             wl_id = reinterpret_cast<uint32_t*>(smem + lay.wl_id);
    float*                wl_d  = reinterpret_cast<float*>(smem + lay.wl_d);
    uint32_t*             nbuf  = reinterpret_cast<uint32_t*>(smem + lay.nb);
    uint64_t*             skey  = reinterpret_cast<uint64_t*>(smem + lay.srt);
    uint64_t*             keys  = reinterpret_cast<uint64_t*>(smem + lay.keys);
    // [0] query, [1] entry distance, then the worklist's length, [4 + 4 p ..] what the
    // worklist tells hop p: first unvisited entry (id, distance), tail distance (as bits:
    // both sides order distances by their bits, a NaN behind +inf);
    // [12 + 4 p ..] candidates in each segment of 32 slots of the hop (kDone: no hop)
    uint32_t*             ctl  = reinterpret_cast<uint32_t*>(smem + lay.ctl);
    uint32_t*             seg  = ctl + 12;
    const uint32_t        R   = a.R;

    for (;;) {
        if (tid == 0) ctl[0] = atomicAdd(a.counter, 1u);
        for (uint32_t w = tid; w < kBloomWords; w += kCtaThreads) bloom[w] = 0u;
        __syncthreads();
        const uint32_t q = ctl[0];
        if (q >= a.nq) break;
        const uint32_t L  = a.Lq != nullptr ? max(1u, min(__ldg(a.Lq + q), a.L)) : a.L;
        const uint32_t kq = a.kq != nullptr ? min(__ldg(a.kq + q), a.k) : a.k;
        const uint32_t entry = a.entry;
        uint32_t       n = 1;  // worklist entries (warp 0)

        if (warp == 0) {
            hop_barrier();  // the entry's distance
            // initializeWorklist: entry visited, distance computed, not in the filter.  Entry
            // e of the list is in lane e % 32, register e / 32: distance bits (kNone past
            // the end) and id | visited.
            uint32_t parent = entry, hops = 0, nv = 0, p = 0;
            float    pd = __uint_as_float(ctl[1]);
            uint32_t e_d  = __float_as_uint(kInf);  // the first unvisited entry, as the others know it
            bool     e_in = false;
            uint32_t wd[LREG], wp[LREG];
#pragma unroll
            for (int r = 0; r < LREG; ++r) {
                wd[r] = kNone;
                wp[r] = kVisitedBit;
            }
            if (lane == 0) {
                wd[0]    = ctl[1];
                wp[0]    = entry | kVisitedBit;
                wl_id[0] = entry | kVisitedBit;
                wl_d[0]  = pd;
                ctl[4]   = kNone;
                ctl[5]   = __float_as_uint(kInf);
                ctl[6]   = L == 1u ? __float_as_uint(pd) : open;
            }
            __syncwarp();
            for (;;) {
                ++hops;
                if (a.vis_ids != nullptr && nv < a.max_visited) {
                    if (lane == 0) {
                        a.vis_ids[(uint64_t)q * a.max_visited + nv] = parent;
                        a.vis_d[(uint64_t)q * a.max_visited + nv]   = pd;
                    }
                    ++nv;
                }
                hop_barrier();  // the hop's distances are there
                const uint32_t* nb_id = nbuf + 2u * SLOTS * p;
                const float*    nb_d  = reinterpret_cast<const float*>(nb_id + SLOTS);

                // the candidates that can enter
                const uint32_t tail = n == L ? __float_as_uint(wl_d[L - 1]) : open;
                uint32_t       kc = 0, best = kNone;
#pragma unroll
                for (int s = 0; s < SPL; ++s) {
                    const uint32_t j    = (uint32_t)s * 32u + lane;
                    const float    dd   = nb_d[j];
                    const uint32_t id   = nb_id[j];
                    const bool     keep = lane < seg[4u * p + s] && __float_as_uint(dd) < tail;
                    const uint32_t m    = __ballot_sync(0xffffffffu, keep);
                    if (keep) {
                        best = min(best, __float_as_uint(dd));
                        skey[kc + __popc(m & ((1u << lane) - 1u))] = make_key(dd, id);
                        // a parent to come: its list into L2
                        for (uint32_t b = 0; b < R; b += 32u) {
                            prefetch_l2(a.adj + (uint64_t)id * R + b);
                            prefetch_l2(a.adj_h + (uint64_t)id * R + b);
                        }
                        prefetch_l2(a.deg + id);
                    }
                    kc += __popc(m);
                }
                __syncwarp();
                if (kc > 32u) {  // several batches below: in (distance, id) order
                    uint64_t key[SPL];
#pragma unroll
                    for (int s = 0; s < SPL; ++s) {
                        const uint32_t j = (uint32_t)s * 32u + lane;
                        key[s]           = j < kc ? skey[j] : ~0ull;
                    }
                    warp_bitonic_sort<SPL>(key, lane);
                    __syncwarp();
#pragma unroll
                    for (int s = 0; s < SPL; ++s) skey[(uint32_t)s * 32u + lane] = key[s];
                    __syncwarp();
                }
                // mergeIntoWorklist by counting: a new entry lands at #(existing at or below
                // its distance) + its rank among the new, an existing one moves down by the
                // new ones strictly closer; the first L stay
                for (uint32_t b0 = 0; b0 < kc; b0 += 32u) {
                    const uint32_t bc = min(32u, kc - b0);
                    const uint64_t cj = lane < bc ? skey[b0 + lane] : ~0ull;
                    uint32_t       at = 0, sh[LREG];
#pragma unroll
                    for (int r = 0; r < LREG; ++r) sh[r] = 0u;
#pragma unroll 2
                    for (uint32_t k = 0; k < bc; ++k) {
                        const uint64_t ck = skey[b0 + k];
                        const uint32_t cd = (uint32_t)(ck >> 32);
                        at += (ck < cj || (ck == cj && k < lane)) ? 1u : 0u;
                        uint32_t before = 0;
#pragma unroll
                        for (int r = 0; r < LREG; ++r) {
                            sh[r] += cd < wd[r] ? 1u : 0u;
                            before += __popc(__ballot_sync(0xffffffffu, wd[r] <= cd));
                        }
                        if (lane == k) at += before;
                    }
#pragma unroll
                    for (int r = 0; r < LREG; ++r) {
                        const uint32_t e = (uint32_t)r * 32u + lane, to = e + sh[r];
                        if (e < n && to < L) {
                            wl_id[to] = wp[r];
                            wl_d[to]  = __uint_as_float(wd[r]);
                        }
                    }
                    if (lane < bc && at < L) {
                        wl_id[at] = (uint32_t)cj;
                        wl_d[at]  = key_dist(cj);
                    }
                    n = min(n + bc, L);
                    __syncwarp();
#pragma unroll
                    for (int r = 0; r < LREG; ++r) {
                        const uint32_t e = (uint32_t)r * 32u + lane;
                        if (e < n) {
                            wp[r] = wl_id[e];
                            wd[r] = __float_as_uint(wl_d[e]);
                        }
                    }
                }
                // the first two unvisited entries: the next parent, which warps 1 .. SPL have
                // chosen already, and what they need for the choice after
                uint32_t u[2] = {kNone, kNone};
#pragma unroll
                for (int r = 0; r < LREG; ++r) {
                    uint32_t m = __ballot_sync(0xffffffffu, !(wp[r] & kVisitedBit));
                    if (m != 0u && u[0] == kNone) {
                        u[0] = 32u * (uint32_t)r + __ffs(m) - 1u;
                        m &= m - 1u;
                    }
                    if (m != 0u && u[1] == kNone) u[1] = 32u * (uint32_t)r + __ffs(m) - 1u;
                }
                // the same rule as theirs, so that both sides stop at the same hop (a new
                // candidate at +inf is no parent)
                best = __reduce_min_sync(0xffffffffu, best);
                if ((!e_in && best >= e_d) || hops >= a.max_hops) break;
                e_in = u[1] != kNone;
                e_d  = __float_as_uint(e_in ? wl_d[u[1]] : kInf);
                parent = wl_id[u[0]];
                pd     = wl_d[u[0]];
                p ^= 1u;
                if (lane == 0) {
                    uint32_t* o = ctl + 4 + 4u * p;
                    *reinterpret_cast<uint4*>(o) =
                        make_uint4(e_in ? wl_id[u[1]] : kNone, e_d, n == L ? __float_as_uint(wl_d[L - 1]) : open, 0u);
                }
#pragma unroll
                for (int r = 0; r < LREG; ++r)
                    if (u[0] == 32u * (uint32_t)r + lane) wp[r] |= kVisitedBit;
                __syncwarp();
            }
            if (lane == 0 && a.vis_n != nullptr) a.vis_n[q] = nv;
            if (lane == 0) ctl[1] = n;
        } else {
            Query<S, DC> qv;
            load_query<S, DC>(qv, a.queries + (uint64_t)q * a.D, a.D, lane, a.center);
            uint32_t skip = kNone;
            if (a.skip_mode == 1) skip = q;
            if (a.skip_mode == 2) skip = a.skip_base + q;
            uint32_t hops = 0, evals = 1, adjw = 0, p = 0, parent = entry;
            // warps 1 .. SPL: each takes the next parent for itself, and the 32 slots of its
            // list that are its segment
            const uint32_t sg   = warp - 1u;
            const bool     ctrl = sg < (uint32_t)SPL;
            const uint32_t slot = 32u * sg + lane;
            uint32_t       nid = 0, hp = 0, dg = 0;
            auto           fetch_row = [&](uint32_t node) {
                nid = slot < R ? __ldg(a.adj + (uint64_t)node * R + slot) : 0u;
                hp  = slot < R ? __ldg(a.adj_h + (uint64_t)node * R + slot) : 0u;
                dg  = __ldg(a.deg + node);
            };
            if (ctrl) fetch_row(entry);
            if (warp == 1) {
                const float d0 =
                    dist_group<S, DC, IQ, M>(qv, a.store, a.scale, [&](int) { return entry; }, 1, a.D, lane);
                if (lane == 0) ctl[1] = __float_as_uint(d0);
            }
            hop_barrier();  // the entry's distance
            for (;;) {
                uint32_t* nb_id = nbuf + 2u * SLOTS * p;
                float*    nb_d  = reinterpret_cast<float*>(nb_id + SLOTS);
                const uint32_t h1 = hp >> 16, h2 = hp & 0xffffu;
                bool           pass = false;
                if (ctrl) {
                    uint32_t c = kDone;
                    if (parent != kNone && hops >= a.max_hops) {
                        if (tid == 32u) atomicOr(a.status, kStatusHopLimit);
                    } else if (parent != kNone) {
                        // filterNeighbors: every slot checks the filter as it stood before
                        // this expansion (the marks follow the barrier)
                        ++hops;
                        dg = dg < R ? dg : R;
                        adjw += dg;
                        pass = slot < dg && nid != skip;
                        // slots past the degree hold whatever was in memory: their filter
                        // slots may lie outside the filter
                        if (pass) pass = !((bloom[h1 >> 5] >> (h1 & 31u)) & (bloom[h2 >> 5] >> (h2 & 31u)) & 1u);
                        if (a.tomb != nullptr && pass) pass = !((__ldg(a.tomb + (nid >> 5)) >> (nid & 31u)) & 1u);
                        const uint32_t m = __ballot_sync(0xffffffffu, pass);
                        if (pass) nb_id[32u * sg + __popc(m & ((1u << lane) - 1u))] = nid;
                        c = __popc(m);
                    }
                    if (lane == 0) seg[4u * p + sg] = c;
                }
                gather_barrier();
                uint32_t c[SPL], cnt = 0;
#pragma unroll
                for (int s = 0; s < SPL; ++s) {
                    c[s] = seg[4u * p + s];
                    cnt += c[s];
                }
                if (c[0] == kDone) break;
                if (pass) {
                    atomicOr(&bloom[h1 >> 5], 1u << (h1 & 31u));
                    atomicOr(&bloom[h2 >> 5], 1u << (h2 & 31u));
                }
                evals += cnt;
                // a quarter of the rows per warp; row j of the hop sits at slot_of(j)
                auto slot_of = [&](uint32_t j) {
                    uint32_t at = j, before = 0;
#pragma unroll
                    for (int s = 0; s + 1 < SPL; ++s) {
                        before += c[s];
                        if (j >= before) at = 32u * (uint32_t)(s + 1) + (j - before);
                    }
                    return at;
                };
                const uint32_t per = (cnt + kCtaGather - 1u) / kCtaGather;
                const uint32_t beg = min(cnt, (warp - 1u) * per), end = min(cnt, beg + per);
                for (uint32_t g0 = beg; g0 < end; g0 += G) {
                    const int      gc = (int)min(G, end - g0);
                    const float    y  = dist_group<S, DC, IQ, M>(
                        qv, a.store, a.scale, [&](int j) { return nb_id[slot_of(g0 + (uint32_t)j)]; }, gc, a.D, lane);
                    const uint32_t vi = round_row_of_lane<S, DC, M>(lane);
                    if (round_writer<S, DC, M>(lane) && (int)vi < gc) nb_d[slot_of(g0 + vi)] = y;
                }
                hop_barrier();  // the distances are there, and the previous merge is done
                if (ctrl) {
                    // next parent: the best candidate that can enter, or the first unvisited
                    // entry, whichever is closer (the entry on equal distance)
                    const uint4 st = *reinterpret_cast<const uint4*>(ctl + 4 + 4u * p);
                    uint32_t    bd = kNone, bi = kNone;
#pragma unroll
                    for (int s = 0; s < SPL; ++s) {
                        const uint32_t j  = (uint32_t)s * 32u + lane;
                        const uint32_t id = nb_id[j], u = __float_as_uint(nb_d[j]);
                        const bool     in = lane < c[s] && u < st.z && (u < bd || (u == bd && id < bi));
                        bd                = in ? u : bd;
                        bi                = in ? id : bi;
                    }
                    const uint32_t md = __reduce_min_sync(0xffffffffu, bd);
                    const uint32_t mi = __reduce_min_sync(0xffffffffu, bd == md ? bi : kNone);
                    parent = mi != kNone && md < st.y ? mi : st.x;
                    if (parent != kNone) fetch_row(parent);
                }
                p ^= 1u;
            }
            if (warp == 1 && lane == 0) {
                if (a.hops_out != nullptr) a.hops_out[q] = hops;
                if (a.evals_out != nullptr) a.evals_out[q] = evals;
                if (a.adjw_out != nullptr) a.adjw_out[q] = adjw;
            }
        }
        __syncthreads();
        n = ctl[1];

        // outputs
        if (a.out_ids != nullptr) {
            if (a.rerank) {
                // exact FP32 distances of the final worklist, sorted (dist, position)
                constexpr int       MF = 4;
                constexpr uint32_t  GF = MF * Layout<StoreF32, DC>::kP;
                Query<StoreF32, DC> qf;
                load_query<StoreF32, DC>(qf, a.queries + (uint64_t)q * a.D, a.D, lane);
                for (uint32_t g0 = warp * GF; g0 < n; g0 += GF * (kCtaThreads / 32u)) {
                    const int      gc = (int)min(GF, n - g0);
                    const float    y  = dist_group<StoreF32, DC, false, MF>(
                        qf, a.vecs_f32, nullptr, [&](int j) { return wl_id[g0 + j] & ~kVisitedBit; }, gc, a.D, lane);
                    const uint32_t vi = round_row_of_lane<StoreF32, DC, MF>(lane);
                    if (round_writer<StoreF32, DC, MF>(lane) && (int)vi < gc) keys[g0 + vi] = make_key(y, g0 + vi);
                }
                __syncthreads();
                for (uint32_t i = tid; i < n; i += kCtaThreads) {
                    const uint64_t key  = keys[i];
                    uint32_t       rank = 0;
                    for (uint32_t k = 0; k < n; ++k) rank += keys[k] < key ? 1u : 0u;
                    if (rank < a.k) {
                        const uint64_t o = (uint64_t)q * a.k + rank;
                        a.out_ids[o]     = rank < kq ? wl_id[i] & ~kVisitedBit : kNone;
                        a.out_d[o]       = rank < kq ? key_dist(key) : kInf;
                    }
                }
                for (uint32_t t = n + tid; t < a.k; t += kCtaThreads) {
                    a.out_ids[(uint64_t)q * a.k + t] = kNone;
                    a.out_d[(uint64_t)q * a.k + t]   = kInf;
                }
            } else {
                for (uint32_t t = tid; t < a.k; t += kCtaThreads) {
                    const uint64_t o  = (uint64_t)q * a.k + t;
                    const bool     in = t < n && t < kq;
                    a.out_ids[o]      = in ? wl_id[t] & ~kVisitedBit : kNone;
                    a.out_d[o]        = in ? wl_d[t] : kInf;
                }
            }
        }
        __syncthreads();
    }
}

template <typename S, int DC, int SPL, int LREG, bool IQ>
static cudaError_t launch_cta_t(const SearchArgs& a, int num_sms, cudaStream_t st) {
    const size_t smem = CtaSearchLayout::make(a.L, SPL * 32, a.rerank != 0).bytes;
    auto         kern = search_cta_kernel<S, DC, SPL, LREG, IQ>;
    cudaError_t  e    = allow_smem(kern, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e          = fit_carveout(kern, kCtaThreads, smem, &per_sm);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    uint64_t grid = (uint64_t)per_sm * num_sms;
    if (grid > a.nq) grid = a.nq;
    if (grid == 0) return cudaSuccess;
    const bool strict = DC == 0 && a.R <= 64 && a.L <= 64;  // the register-worklist kernel's shapes
    kern<<<(unsigned)grid, kCtaThreads, smem, st>>>(a, strict);
    return cudaGetLastError();
}

template <typename S, int DC, bool IQ, int SPL>
static cudaError_t launch_cta_spl(const SearchArgs& a, int num_sms, cudaStream_t st) {
    if (a.L <= 64) return launch_cta_t<S, DC, SPL, 2, IQ>(a, num_sms, st);
    if (a.L <= 128) return launch_cta_t<S, DC, SPL, 4, IQ>(a, num_sms, st);
    return launch_cta_t<S, DC, SPL, 8, IQ>(a, num_sms, st);
}

template <typename S, int DC, bool IQ = false>
static cudaError_t launch_cta(const SearchArgs& a, int num_sms, cudaStream_t st) {
    if (a.R <= 64) return launch_cta_spl<S, DC, IQ, 2>(a, num_sms, st);
    return launch_cta_spl<S, DC, IQ, 4>(a, num_sms, st);
}

}  // namespace vann
