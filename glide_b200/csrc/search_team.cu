// Search kernels that give a query a CTA instead of a warp, for batches that leave the device idle
// otherwise (TeamCall in beam_core.cuh).
#include "search_core.cuh"

namespace glide {

namespace {

constexpr uint32_t kMaxScoring = 8;   // warps of a team that score, with or without the master

template<int NB, int NC, bool LANES, bool PARTS, typename D>
__global__ void __launch_bounds__((kMaxScoring + 1) * 32, NB <= 2 ? 3 : 2) search_team_kernel(const SearchDev d) {
    search_body<NB, NC, LANES, PARTS, true>(d, D{d.a.dim});
}

// Which team size: as many scoring warps as an expansion has batches for (eight rows a warp, four of wide ones),
// as long as every query of the batch has its CTA resident at once; with half of them before a warp per query
// (0) is the better form. Search kernel, us, a warp per query against teams of so many warps:
//   128 values, degree 32, beam 64    one query 207, 3: 149, 5: 120; 600 queries 354, 3: 236, 5: 187; 1,250: 371, 3: 272,
//                                     5 (not all resident): 348; 1,600 (3 not all resident): 387, 3: 444
//   100 values, degree 32, beam 128   one query 416, 5: 227; 600 queries 667, 3: 438, 5 (not all resident): 593
//   960 values, degree 64, beam 64    one query 600, 2: 441, 4: 316, 8: 242; 600: 680, 2: 448, 4: 350, 8 (not all): 491;
//                                     2,000: 832, 2: 727, 4 (not all): 795
// In a device that is full a team loses: the master's turns leave its other warps waiting.
uint32_t team_warps(const void *kernel, const SearchArgs &a, size_t smem_bytes, int sms) {
    const bool fit = rows_fit_lanes(a.dim);
    const uint32_t rows = fit ? 8u : (uint32_t) kWideRows, alone = fit ? 1u : 0u;   // the master scores wide rows only
    uint32_t scoring = kMaxScoring;
    while (scoring > 2 && (scoring / 2) * rows >= a.degree) scoring >>= 1;
    for (; scoring >= 2; scoring >>= 1) {
        int per_sm = 0;
        const uint32_t warps = scoring + alone;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, (int) warps * 32, smem_bytes) != cudaSuccess) return 0;
        if ((uint64_t) per_sm * (uint64_t) sms >= a.Q) return warps;
    }
    return 0;
}

template<int NB, int NC, bool LANES, typename D>
void (*team_instance(const SearchArgs &a))(const SearchDev) {
    if constexpr (NB > 1) {
        if (a.parts != nullptr) return search_team_kernel<NB, NC, LANES, true, D>;
    }
    return search_team_kernel<NB, NC, LANES, false, D>;
}

template<int NB, int NC, bool LANES>
cudaError_t launch_team_t(const SearchDev &given, size_t smem_bytes, int sms, cudaStream_t stream, uint32_t *team_warps_out) {
    SearchDev d = given;
    void (*kernel)(const SearchDev) = rows_fit_lanes(d.a.dim) ? team_instance<NB, NC, LANES, DimOf<true>>(d.a) : team_instance<NB, NC, LANES, DimOf<false>>(d.a);
    if (smem_bytes > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem_bytes);
        if (e != cudaSuccess) return e;
    }
    const uint32_t warps = team_warps(reinterpret_cast<const void *>(kernel), d.a, smem_bytes, sms);
    if (warps == 0) return cudaSuccess;
    d.a.ticket = nullptr;   // every query has its CTA
    kernel<<<d.a.Q, warps * 32, smem_bytes, stream>>>(d);
    *team_warps_out = warps;
    return cudaGetLastError();
}

}  // namespace

template<typename D>
static void preload_team_instances(const SearchDev &d, cudaStream_t stream) {
    const size_t call = sizeof(TeamCall);   // all that the master's farewell to its helper touches
    search_team_kernel<1, 2, true, false, D><<<1, 64, call, stream>>>(d);
    search_team_kernel<2, 2, true, false, D><<<1, 64, call, stream>>>(d);
    search_team_kernel<4, 2, true, false, D><<<1, 64, call, stream>>>(d);
    search_team_kernel<2, 2, false, false, D><<<1, 64, call, stream>>>(d);
}

// The instances that small batches take, as preload_search_kernels: Q = 0, the master quits at once.
void preload_search_team_kernels(cudaStream_t stream) {
    const SearchDev d{};
    preload_team_instances<DimOf<true>>(d, stream);
    preload_team_instances<DimOf<false>>(d, stream);
}

// Beams above 256 slots and adjacency rows above 64 entries stay with a warp per query (their merges and sorts use
// per-warp scratch of another layout), and so does the streamed large path, which skips most of its queries.
cudaError_t launch_search_team(const SearchArgs &a, cudaStream_t stream, uint32_t *team_warps_out) {
    *team_warps_out = 0;
    if (a.p.beam > 256 || a.degree > 64 || (a.segment_ids != nullptr && a.parts == nullptr)) return cudaSuccess;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    if (a.Q > 32u * (uint32_t) sms) return cudaSuccess;   // more than fit with two warps each (64 warps an SM)
    SearchDev d;
    d.a = a;
    d.max_centroid = pow2_at_least(a.C, 32);
    d.max_topk = a.top_k <= 32 ? 32 : (a.top_k <= 64 ? 64 : 128);
    const uint32_t extra = a.segment_ids ? 4 * d.max_topk : 0;
    d.strip_words = kTeamCallWords + ((strip_words_base(a.dim, 64, a.p.hash_bit) + extra + 3u) & ~3u);
    const size_t bytes = (size_t) d.strip_words * 4;
    if (bytes > 200 * 1024) return cudaSuccess;   // refused by the other form too
    if (a.degree <= 32) {
        if (a.p.beam <= 32 && a.parts == nullptr) return launch_team_t<1, 2, true>(d, bytes, sms, stream, team_warps_out);
        if (a.p.beam <= 64) return launch_team_t<2, 2, true>(d, bytes, sms, stream, team_warps_out);
        if (a.p.beam <= 128) return launch_team_t<4, 2, true>(d, bytes, sms, stream, team_warps_out);
        return launch_team_t<8, 2, true>(d, bytes, sms, stream, team_warps_out);
    }
    if (a.p.beam <= 64) return launch_team_t<2, 2, false>(d, bytes, sms, stream, team_warps_out);
    if (a.p.beam <= 128) return launch_team_t<4, 2, false>(d, bytes, sms, stream, team_warps_out);
    return launch_team_t<8, 2, false>(d, bytes, sms, stream, team_warps_out);
}

}  // namespace glide
