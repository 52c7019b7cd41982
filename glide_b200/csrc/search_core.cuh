// A query's search from its start point to its result rows, shared by the kernels that give a search one
// warp (search.cu) and those that give it a CTA (search_team.cu).
#pragma once

#include "beam_core.cuh"
#include "kernels.h"

namespace glide {

namespace {

struct SearchDev {
    SearchArgs a;
    uint32_t max_centroid;
    uint32_t max_topk;
    uint32_t strip_words;
};

// Last bitonic phase on a shared array of 32*n pairs (the input must be bitonic).
__device__ inline void warp_merge_final_smem(float *k, uint32_t *v, uint32_t n_per_lane) {
    const uint32_t total = 32u * n_per_lane, lane = lane_id();
    for (uint32_t stride = total >> 1; stride >= 1; stride >>= 1) {
        for (uint32_t p = lane; p < total / 2; p += 32) {
            const uint32_t lo = ((p / stride) * 2 * stride) + (p % stride);
            const uint32_t hi = lo + stride;
            const float k0 = k[lo], k1 = k[hi];
            if ((k0 != k1) && !(k0 < k1)) {
                k[lo] = k1; k[hi] = k0;
                const uint32_t t = v[lo]; v[lo] = v[hi]; v[hi] = t;
            }
        }
        __syncwarp();
    }
}

// LANES: adjacency rows of at most 32 entries, candidates stay in registers (beam_loop_lanes);
// the strip then holds only the query and the visited set.
// The partition a large-path search runs in.
struct PartView {
    const float *data;
    const uint32_t *graph, *map;
    uint32_t start_point;
};

template<int NB, int NC, bool LANES, bool PARTS, bool TEAM, typename D>
__device__ __forceinline__ void search_one(const SearchDev &d, const WarpStrip &s, const BeamParams &p, D dim, uint32_t q,
                                           const PartView &given, bool check_routed) {
    const SearchArgs &a = d.a;
    const uint32_t lane = lane_id();
    // outside the multi-partition kernel the partition is the launch's own (kernel parameters, no registers)
    const PartView view = PARTS ? given : PartView{a.data, a.graph, a.map, a.start_point};

    const bool sub = (a.segment_ids != nullptr);
    if (sub && check_routed) {  // search_kernel.cuh:676-692: skip queries not routed to this partition
        bool routed = false;
        if (lane == 0) {
            for (uint32_t i = 0; i < a.segment_num; i++) {
                const uint32_t sid = a.segment_ids[(uint64_t) q * a.segment_num + i];
                if (sid == a.segment_id) { routed = true; break; }
                if (sid == kInvalid) break;
            }
        }
        routed = __shfl_sync(kFullMask, routed ? 1 : 0, 0) != 0;
        if (!routed) return;
    }

    load_query(s.query, a.queries + (uint64_t) q * a.dim, a.dim);
    visited_clear(s.visited, p.hash_bit);
    __syncwarp();

    uint32_t rows = 0;
    uint32_t start_node;
    if (!sub) {
        // the nearest centroid was found by the routing pre-pass (search_kernel.cuh:258-269)
        const uint32_t r = a.route[q];
        start_node = a.start_points[r < a.C ? r : 0u];   // the routing kernels never write an id beyond C; checked all the same
    } else {
        start_node = view.start_point;
    }
    float bk[NB];
    uint32_t bv[NB];
    uint32_t iters;
    if constexpr (LANES) {
        float ck;
        uint32_t cv;
        rows += seed_lanes<TEAM>(s, start_node, kInvalid, view.graph, a.degree, p.hash_bit, view.data, dim, a.metric, ck, cv);
        iters = beam_loop_lanes<NB, TEAM>(bk, bv, s, p, kInvalid, view.graph, a.degree, view.data, dim, a.metric, &rows, ck, cv);
    } else {
        rows += seed_from_row<TEAM>(s, start_node, kInvalid, view.graph, a.degree, p.hash_bit, view.data, dim, a.metric);
        iters = beam_loop<NB, NC, false, TEAM>(bk, bv, s, p, kInvalid, view.graph, a.degree, view.data, dim, a.metric, &rows);
    }

    if (!sub) {
#pragma unroll
        for (int i = 0; i < NB; i++) {
            const uint32_t j = NB * lane + i;
            if (j < a.top_k) {
                a.out_ids[(uint64_t) q * a.top_k + j] = bv[i] & kClean;
                a.out_dists[(uint64_t) q * a.top_k + j] = bk[i];
            }
        }
    } else {
        // result_merge (search_kernel.cuh:609-651): fold the first top_k beam entries
        // into the running result with a network of width max_topk.
        const uint32_t M = d.max_topk, n = M / 32;
        float *mk = reinterpret_cast<float *>(s.extra);
        uint32_t *mv = s.extra + M;
        float *rk = reinterpret_cast<float *>(s.extra + 2 * M);  // this partition's result, by beam position
        uint32_t *rv = s.extra + 3 * M;
#pragma unroll
        for (int i = 0; i < NB; i++) {
            const uint32_t j = NB * lane + i;
            if (j < a.top_k) {
                rk[j] = bk[i];
                const uint32_t id = bv[i] & kClean;
                rv[j] = (id == kPadClean) ? kInvalid : view.map[id];  // an unfilled slot has no global id
            }
        }
        float *fd = a.out_dists + (uint64_t) q * a.top_k;
        uint32_t *fi = a.out_ids + (uint64_t) q * a.top_k;
        for (uint32_t j = lane; j < M; j += 32) {
            mk[j] = (j < a.top_k) ? fd[j] : FLT_MAX;
            mv[j] = (j < a.top_k) ? fi[j] : kInvalid;
        }
        __syncwarp();
        for (uint32_t j = lane; j < M; j += 32) {
            const uint32_t k = M - 1 - j;
            if (k < a.top_k && mk[j] > rk[k]) {
                mk[j] = rk[k];
                mv[j] = rv[k];
            }
        }
        __syncwarp();
        warp_merge_final_smem(mk, mv, n);
        for (uint32_t j = lane; j < a.top_k; j += 32) {
            fd[j] = mk[j];
            fi[j] = mv[j];
        }
    }
    if (a.counters && lane == 0) {
        atomicAdd(a.counters + 0, (unsigned long long) rows);
        atomicAdd(a.counters + 1, (unsigned long long) iters);
        // a team's calls read whole adjacency rows where the rows fit the lanes (team_expand): what they read beside `rows`
        if (TEAM && dim_fits(dim)) atomicAdd(a.counters + 2, (unsigned long long) (iters + 1u) * a.degree - rows);
    }
}

// One query of the launch. PARTS: every partition it is routed to, in ascending partition order: the order
// in which the reference's loop over partitions (glide_large_impl.cuh:424-493) folds them into the running
// result. The routed list is a prefix of the query's row of segment_ids.
template<int NB, int NC, bool LANES, bool PARTS, bool TEAM, typename D>
__device__ __forceinline__ void search_query(const SearchDev &d, const WarpStrip &s, const BeamParams &p, D dim, uint32_t q) {
    const SearchArgs &a = d.a;
    if constexpr (!PARTS) {
        search_one<NB, NC, LANES, false, TEAM>(d, s, p, dim, q, PartView{a.data, a.graph, a.map, a.start_point}, true);
    } else {
        const uint32_t lane = lane_id();
        const uint32_t *ids = a.segment_ids + (uint64_t) q * a.segment_num;
        const uint32_t r0 = lane < a.segment_num ? ids[lane] : kInvalid;
        const uint32_t r1 = lane + 32u < a.segment_num ? ids[lane + 32u] : kInvalid;
        const bool longer = a.segment_num > 64u && ids[64] != kInvalid;   // rare: more than 64 partitions routed
        uint32_t prev = kInvalid;
        while (true) {
            uint32_t best = kInvalid;
            if (r0 != kInvalid && (prev == kInvalid || r0 > prev)) best = r0;
            if (r1 != kInvalid && (prev == kInvalid || r1 > prev) && r1 < best) best = r1;
            if (longer)
                for (uint32_t i = 64u + lane; i < a.segment_num; i += 32u) {
                    const uint32_t sid = ids[i];
                    if (sid != kInvalid && (prev == kInvalid || sid > prev) && sid < best) best = sid;
                }
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) best = min(best, __shfl_xor_sync(kFullMask, best, off));
            if (best == kInvalid) break;
            prev = best;
            const PartitionRef ref = a.parts[best];
            if (ref.data != nullptr) search_one<NB, NC, LANES, true, TEAM>(d, s, p, dim, q, PartView{ref.data, ref.graph, ref.map, ref.start_point}, false);
            __syncwarp();
        }
    }
}

// A warp per query (TEAM: a CTA per query, see TeamCall). With a ticket counter the grid is sized to what
// the device holds at once and every warp draws its next query as soon as it finishes one, so a slow query
// delays neither the other warps of its CTA nor a whole wave of CTAs.
template<int NB, int NC, bool LANES, bool PARTS, bool TEAM, typename D>
__device__ __forceinline__ void search_body(const SearchDev &d, D dim) {
    extern __shared__ __align__(16) uint32_t smem[];
    const SearchArgs &a = d.a;
    const uint32_t searches = TEAM ? 1u : blockDim.x >> 5;   // of a CTA at a time
    const uint32_t warp = threadIdx.x >> 5, lane = lane_id();
    const BeamParams p{a.p.beam, a.p.max_iterations, a.p.min_iterations, a.p.hash_bit, a.p.hash_reset_interval};
    WarpStrip s = make_strip(smem + (TEAM ? kTeamCallWords : (size_t) warp * d.strip_words), a.dim, LANES && !TEAM ? kLaneScratch : 32u * NC, p.hash_bit);
    if constexpr (NB == 16) s.tail = smem + (size_t) (warp + 1) * d.strip_words - kTwoWarpScratch;
    if constexpr (TEAM) {
        s.team = reinterpret_cast<TeamCall *>(smem);
        if (warp != 0) {
            team_serve(s, dim, a.degree, a.metric);
            return;
        }
    }
    if (a.ticket == nullptr) {
        const uint32_t q = blockIdx.x * searches + (TEAM ? 0u : warp);
        if (q < a.Q) search_query<NB, NC, LANES, PARTS, TEAM>(d, s, p, dim, a.order ? a.order[q] : q);
    } else {
        while (true) {
            uint32_t q = 0;
            if (lane == 0) q = atomicAdd(a.ticket, 1u);
            q = __shfl_sync(kFullMask, q, 0);
            if (q >= a.Q) break;
            search_query<NB, NC, LANES, PARTS, TEAM>(d, s, p, dim, a.order ? a.order[q] : q);
            __syncwarp();
        }
    }
    if constexpr (TEAM) team_quit(s);
}

inline uint32_t pow2_at_least(uint32_t x, uint32_t lo) {
    uint32_t m = lo;
    while (m < x) m <<= 1;
    return m;
}

// Grid of a launch: with a ticket counter what the device holds at once, the counter set to zero.
inline cudaError_t search_grid(const void *kernel, const SearchArgs &a, uint32_t ctas, uint32_t threads, size_t smem_bytes, cudaStream_t stream,
                               uint32_t *grid) {
    *grid = ctas;
    if (!a.ticket) return cudaSuccess;
    int per_sm = 0, dev = 0, sms = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, (int) threads, smem_bytes);
    if (e != cudaSuccess) return e;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    const uint32_t resident = (uint32_t) (per_sm > 0 ? per_sm : 1) * (uint32_t) sms;
    if (ctas > resident) *grid = resident;
    return cudaMemsetAsync(a.ticket, 0, sizeof(uint32_t), stream);
}

}  // namespace

}  // namespace glide
