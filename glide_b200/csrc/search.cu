// Query search kernels: the small path's routed search (reference search_kernel,
// search_kernel.cuh:393-490), the large path's query routing (select_segment_kernel,
// :546-607) and per-partition search with running top-k merge (search_on_sub_kernel +
// result_merge, :609-765).
#include <cstdlib>

#include "search_core.cuh"

namespace glide {

namespace {

// Register targets per beam class (measured): 64 registers for beams up to 64 slots (4 CTAs per
// SM), 80 up to 128, 128 beyond. The 32-slot instance does best with the compiler's own choice.
template<int NB, int NC, bool LANES, typename D>
__global__ void __launch_bounds__(256, NB == 2 ? ctas_per_sm<D>(4, 3) : (NB == 4 ? 3 : 2)) search_kernel(const SearchDev d) {
    search_body<NB, NC, LANES, false, false>(d, D{d.a.dim});
}

// 32-slot beams: nine warps per CTA and four CTAs per SM (56 registers) hold 36 queries per SM at
// once, 5,328 on 148 SMs, so that a batch of 10,000 queries is two full rounds; with eight warps
// (4,736 at once) the same batch is two rounds and a third with a tenth of the warps busy.
template<int NC, bool LANES, typename D>
__global__ void __launch_bounds__(288, ctas_per_sm<D>(4, 3)) search_kernel_32(const SearchDev d) {
    search_body<1, NC, LANES, false, false>(d, D{d.a.dim});
}

// select_segment_kernel (search_kernel.cuh:546-607): a warp per query.
__global__ void __launch_bounds__(128) select_segment_kernel(const SelectSegmentArgs a, uint32_t max_centroid,
                                                             uint32_t strip_words) {
    extern __shared__ __align__(16) uint32_t smem[];
    const uint32_t warp = threadIdx.x >> 5, lane = lane_id();
    const uint32_t q = blockIdx.x * (blockDim.x >> 5) + warp;
    if (q >= a.Q) return;
    uint32_t *base = smem + (size_t) warp * strip_words;
    float *query = reinterpret_cast<float *>(base);
    uint32_t *scratch = base + dim_pad4(a.dim);
    load_query(query, a.queries + (uint64_t) q * a.dim, a.dim);
    nearest_centroid(query, a.centroids, a.C, max_centroid, a.dim, a.metric, scratch, kSorted);
    const float *ck = reinterpret_cast<const float *>(scratch);
    const uint32_t *cv = scratch + max_centroid;
    uint32_t *out = a.out + (uint64_t) q * a.C;
    const float d0 = ck[0];
    uint32_t allow_num = 0;
    for (uint32_t base_i = 0; base_i < a.C; base_i += 32) {
        const uint32_t i = base_i + lane;
        const bool allow = (i < a.C) && (ck[i] / d0 <= a.boundary_factor);
        if (i < a.C) out[i] = allow ? cv[i] : kInvalid;
        allow_num += __popc(__ballot_sync(kFullMask, allow));
    }
    __syncwarp();
    if (allow_num < a.min_segment_num) {
        const uint32_t need = a.min_segment_num - allow_num;
        for (uint32_t i = lane; i < need; i += 32)
            if (allow_num + i < a.C) out[allow_num + i] = cv[allow_num + i];
    }
}

// Large path with every partition in device memory: a warp walks all the partitions its query is routed to.
template<int NB, int NC, bool LANES, typename D>
__global__ void __launch_bounds__(256, NB <= 2 ? 3 : (NB == 4 ? ctas_per_sm<D>(3, 2) : 2)) search_parts_kernel(const SearchDev d) {
    search_body<NB, NC, LANES, true, false>(d, D{d.a.dim});
}

template<int NB, int NC, bool LANES, typename D>
void (*search_instance(const SearchArgs &a))(const SearchDev) {
    if constexpr (NB == 1) return search_kernel_32<NC, LANES, D>;
    else return a.parts != nullptr ? search_parts_kernel<NB, NC, LANES, D> : search_kernel<NB, NC, LANES, D>;
}

template<int NB, int NC, bool LANES = false>
cudaError_t launch_search_t(const SearchDev &d, uint32_t warps_per_cta, size_t smem_bytes, cudaStream_t stream) {
    void (*kernel)(const SearchDev);
    if constexpr (NC == 2) kernel = rows_fit_lanes(d.a.dim) ? search_instance<NB, NC, LANES, DimOf<true>>(d.a) : search_instance<NB, NC, LANES, DimOf<false>>(d.a);
    else kernel = search_instance<NB, NC, LANES, uint32_t>(d.a);   // adjacency rows above 64 entries
    if (smem_bytes > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem_bytes);
        if (e != cudaSuccess) return e;
    }
    uint32_t grid = 0;
    cudaError_t e = search_grid(reinterpret_cast<const void *>(kernel), d.a, (d.a.Q + warps_per_cta - 1) / warps_per_cta, warps_per_cta * 32, smem_bytes, stream, &grid);
    if (e != cudaSuccess) return e;
    kernel<<<grid, warps_per_cta * 32, smem_bytes, stream>>>(d);
    return cudaGetLastError();
}

}  // namespace

// See preload_build_kernels: launches without work (Q = 0, no ticket) that load the common instances, for rows that fit
// the lanes and for others.
template<typename D>
static void preload_search_instances(const SearchDev &d, cudaStream_t stream) {
    search_kernel_32<2, true, D><<<1, 32, 0, stream>>>(d);
    search_kernel<2, 2, true, D><<<1, 32, 0, stream>>>(d);
    search_kernel<4, 2, true, D><<<1, 32, 0, stream>>>(d);
    search_kernel<2, 2, false, D><<<1, 32, 0, stream>>>(d);
}

cudaError_t preload_search_kernels(cudaStream_t stream) {
    const SearchDev d{};
    preload_search_instances<DimOf<true>>(d, stream);
    preload_search_instances<DimOf<false>>(d, stream);
    preload_search_team_kernels(stream);
    return cudaGetLastError();
}

cudaError_t launch_search(const SearchArgs &a, cudaStream_t stream, uint32_t *team_warps) {
    uint32_t team = 0;
    if (team_warps) *team_warps = 0;
    if (a.Q == 0) return cudaSuccess;
    const cudaError_t te = launch_search_team(a, stream, &team);
    if (team_warps) *team_warps = team;
    if (te != cudaSuccess || team) return te;
    SearchDev d;
    d.a = a;
    d.max_centroid = pow2_at_least(a.C, 32);
    d.max_topk = a.top_k <= 32 ? 32 : (a.top_k <= 64 ? 64 : 128);  // kernel_config.cuh:309-319
    // same size ladders as kernel_config.cuh:190-204 so that ties fall identically
    const uint32_t max_beam = a.p.beam <= 64 ? 64 : (a.p.beam <= 128 ? 128 : (a.p.beam <= 256 ? 256 : 512));
    const uint32_t max_cand = a.degree <= 64 ? 64 : (a.degree <= 128 ? 128 : 256);
    const uint32_t extra = a.segment_ids ? 4 * d.max_topk : 0;
    const bool lanes = a.degree <= 32;
    d.strip_words = (strip_words_base(a.dim, lanes ? kLaneScratch : max_cand, a.p.hash_bit) + extra + two_warp_scratch_words(max_beam) + 3u) & ~3u;
    const size_t strip_bytes = (size_t) d.strip_words * 4;
    uint32_t warps = 8;
    while (warps > 1 && strip_bytes * warps > 96 * 1024) warps >>= 1;
    if (strip_bytes * warps > 200 * 1024) return cudaErrorInvalidValue;
    const int nb = max_beam / 32, nc = max_cand / 32;
    if (lanes) {
        if (a.p.beam <= 32 && warps == 8 && strip_bytes * 9 * 4 <= 200 * 1024 && a.parts == nullptr) {
            static const uint32_t w32 = [] {   // experiments: GLIDE_B200_SEARCH_WARPS=8 restores eight warps per CTA
                const char *e = std::getenv("GLIDE_B200_SEARCH_WARPS");
                const uint32_t v = e ? (uint32_t) std::strtoul(e, nullptr, 10) : 9u;
                return (v >= 1 && v <= 9) ? v : 9u;
            }();
            warps = w32;
        }
        const size_t bytes = strip_bytes * warps;
        if (a.p.beam <= 32 && a.parts == nullptr) return launch_search_t<1, 2, true>(d, warps, bytes, stream);   // (the 64-slot kernel gives the same beam)
        if (nb == 2) return launch_search_t<2, 2, true>(d, warps, bytes, stream);
        if (nb == 4) return launch_search_t<4, 2, true>(d, warps, bytes, stream);
        if (nb == 8) return launch_search_t<8, 2, true>(d, warps, bytes, stream);
        return launch_search_t<16, 2, true>(d, warps, bytes, stream);
    }
    GLIDE_DISPATCH_NB_NC(launch_search_t, nb, nc, d, warps, strip_bytes * warps, stream);
}

cudaError_t launch_select_segments(const SelectSegmentArgs &a, cudaStream_t stream) {
    if (a.Q == 0) return cudaSuccess;
    const uint32_t max_centroid = pow2_at_least(a.C, 32);
    const uint32_t strip_words = (dim_pad4(a.dim) + 2 * max_centroid + 3u) & ~3u;
    const uint32_t warps = 4;
    const size_t smem_bytes = (size_t) strip_words * 4 * warps;
    if (smem_bytes > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(select_segment_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int) smem_bytes);
        if (e != cudaSuccess) return e;
    }
    select_segment_kernel<<<(a.Q + warps - 1) / warps, warps * 32, smem_bytes, stream>>>(a, max_centroid, strip_words);
    return cudaGetLastError();
}

}  // namespace glide
