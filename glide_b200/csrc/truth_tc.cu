// Exact brute-force kNN on the tensor cores: ground truth for large query or base sets. What comes out is
// what bruteforce_tile_kernel gives bit for bit: the tensor cores only decide which rows are looked at.
//
//   norms      |b|^2 of every base row, and the largest |b| and |b - tf32(b)|.
//   contract   a CTA owns 128 queries and every slices-th tile of 128 base rows. Operand blocks of 32 values
//              arrive by TMA (128-byte swizzle) into a ring of shared-memory stages; the queries' blocks stay
//              in shared memory where they fit (up to 256 values a row), otherwise they ride along with the
//              rows'. tcgen05.mma kind::tf32 accumulates the 128 x 128 dot products in tensor memory (two
//              buffers), sixteen epilogue warps turn them into a = |b|^2 - 2 q.b (thread (query, part): 32 columns).
//   threshold  a pass over every stride-th row keeps minima over groups of rows that lie tiles apart (neighbours in the file
//              are often neighbours in space; a group has few of a query's k nearest rows even where the file is sorted by
//              cluster); the k-th smallest of them, t, is an upper bound of the k-th smallest a. The true k nearest then have
//              a <= t + 2E, where E bounds |a + |q|^2 - d| for the fp32 distance d: tf32 rounding by Cauchy's inequality from
//              the norms of what it drops, which is nothing for integers below 2048; sums by their length, four steps of 2^-23
//              a term (how the tensor core accumulates is not specified: an assumption, and a generous one).
//   select     the pass over all tiles stores every column with a <= t + 2E.
//   re-rank    their fp32 distances in the order of bruteforce_tile_kernel, sorted by (distance, id).
//
// A query with more candidates than its buffer holds (foreseen from the sample where it can be), or fewer than k, or with values
// beyond the bounds, is left to bruteforce_tile_kernel, in the segment form with the 63 rows beside it to segment_knn_kernel; a
// tensor map that cannot be made or a wait that runs out leaves everything to them. Where it is the norms that make most rows
// candidates, a second attempt takes rows and queries about a point amid them.
// Bound by the epilogue's chain per tile and the trip of the row tiles from L2 (once per 128 queries): the select pass over 1M x
// 128 rows for 1,000 queries takes 0.82 ms, its 256 GFLOP are 0.31 ms at half of the measured bf16 rate.
// bruteforce_tile_kernel against this: 1M x 128 rows, 1,000 queries, k = 10: 22.7 to 1.12 ms, k = 100: 39.1 to 2.34 ms; 100,000 x
// 960, 333 queries 6.5 to 0.58 ms; 1M x 64, 10 queries 1.79 to 0.27 ms; 4,000 x 32, 10 queries 122 to 72 us; 300,000 x 96 in
// clusters of 1,000 one after another, 1,000 queries, k = 100: 31.7 to 5.9 ms; 50,000 x 64 around 1,000, 100 queries 392 to
// 182 us. 5,000 equal rows, 100 queries 729 to 819 us: an attempt is lost.
#include <algorithm>
#include <vector>

#include "common.cuh"
#include "kernels.h"
#include "umma.cuh"

namespace glide {

namespace {

using namespace umma;

constexpr uint32_t kTile = 128;              // queries per CTA, base rows per tile
constexpr uint32_t kBlock = 32;              // values of a row per operand block
constexpr uint32_t kBlockBytes = kTile * kBlock * 4;
constexpr uint32_t kParts = 4;               // epilogue threads per query
constexpr uint32_t kEpi = 4 * kParts;        // epilogue warps
constexpr uint32_t kTruthThreads = (kEpi + 2) * 32;
constexpr uint32_t kResidentBlocks = 8;      // query blocks kept in shared memory
constexpr uint32_t kCap = 3968;              // candidates per query; with up to 128 earlier results 4,096 sort keys
constexpr uint32_t kSegCap = 2048;           // candidates per row of a segment call
constexpr uint32_t kSegRows = 1u << 21;      // rows of the largest partition of a segment call

// Largest |b|^2 and |b - tf32(b)|^2 of the base rows (of a partition), as bits: non-negative floats order as integers.
struct TruthTops {
    uint32_t norm, rest;
};

// Rows whose |b|^2 is no number below this are nobody's neighbour as long as the k-th smallest a is below kFarBound and
// |q|^2 below kFarQuery: a >= |b| (|b| - 2 |q|) > 9e35 for them. Their norm is set to infinity, so that they meet no threshold,
// and they count in no bound.
constexpr float kFarNorm = 1e36f, kFarBound = 1e34f, kFarQuery = 1e32f;

// What the call hands back: queries, or (segment form) halves of 64 rows of a tile, that have too many candidates, too few, or
// values beyond the bounds. A query's `thr` is then -infinity: later kernels pass it by.
struct TruthBad {
    uint32_t *gave_up;                       // a wait ran out: everything
    uint32_t *count, *items;
    uint32_t *hopeful;                       // queries handed back that the error bound alone, not the rows, gave too many candidates
    uint32_t *seen;                          // segment form: one flag per half, each is listed once
    uint32_t first;                          // added to the queries of a pass
};

// A CTA's share of a partition's own kNN graph (segment form): rows [first, first + 128) of the partition are the
// queries, all of its rows the base; `stride`, `span` and `runs` are the sample's, as in TruthArgs.
struct SegmentTile {
    uint32_t seg_start, seg_len, first, stride, span, runs, part, index;
};

struct TruthArgs {
    uint32_t n, Q, dim, kblocks, stages, cap;
    uint32_t map_from;                       // the tensor maps' first row
    bool give_up;                            // as if a wait had run out
    const SegmentTile *segments;             // segment form: one per CTA; per-query arrays are indexed by CTA * 128 + row
    uint32_t slices;                         // CTA (query tile, slice) takes tiles slice, slice + slices, ...
    // sample pass: column c stands for row c * stride; a thread keeps the minima of its columns over `span` of its tiles,
    // takes the minimum of every `fold` of them and stores those, for each of `runs` such spans; `groups` minima per query
    uint32_t stride, span, runs, fold, groups;
    const float *norms;
    const float *thr;                        // per query (select pass)
    float *gmin;                             // Q x groups
    uint32_t *count;                         // per query
    uint32_t *cand;                          // Q x cap
    uint32_t *gave_up;
};

__device__ __forceinline__ void report_bad(const TruthBad &bad, uint32_t item) {
    if (bad.seen == nullptr || atomicExch(bad.seen + item, 1u) == 0u) bad.items[atomicAdd(bad.count, 1u)] = bad.first + item;
}

__device__ __forceinline__ float tf32_rest(float x) { return x - __uint_as_float(__float_as_uint(x) & 0xffffe000u); }

// The point that rows are taken about in a second attempt (TcLeft): the mean of up to 64 rows, evenly spaced, of a call's base or
// (segment form, in the CTAs of its first tile) of a partition.
__global__ void __launch_bounds__(128) truth_centre_kernel(const float *__restrict__ data, uint32_t rows, uint32_t dim, const SegmentTile *__restrict__ segments,
                                                           float *centre) {
    if (segments != nullptr) {
        const SegmentTile t = segments[blockIdx.y];
        if (t.first != 0) return;
        data += (uint64_t) t.seg_start * dim;
        rows = t.seg_len;
        centre += (uint64_t) t.part * dim;
    }
    const uint32_t d = blockIdx.x * 128u + threadIdx.x, count = min(rows, 64u);
    if (d >= dim) return;
    float sum = 0.0f, used = 0.0f;
    for (uint32_t i = 0; i < count; i++) {
        const float v = __ldg(data + (uint64_t) i * rows / count * dim + d);
        if (fabsf(v) < 1e18f) {
            sum += v;
            used += 1.0f;
        }
    }
    centre[d] = used > 0.0f ? sum / used : 0.0f;
}

// A warp per row: |x|^2, |x - tf32(x)|^2 (two floats per row if `rest` is given) and the maxima. Segment form: a CTA per tile,
// maxima per partition. Not kRowsInPlace: the rows padded to `pitch` are written too, from row `padded_from` on; kRowsCentred: x is
// the row less a centre (one per partition); what the subtraction rounds off is far within the bound on the sums.
enum RowsForm : int { kRowsInPlace = 0, kRowsPadded = 1, kRowsCentred = 2 };
template<int FORM>
__global__ void __launch_bounds__(256, 8) truth_rows_kernel(const float *__restrict__ data, uint32_t rows, uint32_t dim, float *norms, float *rest,
                                                            uint32_t pitch, float *padded, uint32_t padded_from, TruthTops *tops,
                                                            const SegmentTile *__restrict__ segments, const float *__restrict__ centre) {
    __shared__ uint32_t top[2];
    if (threadIdx.x < 2) top[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t lane = lane_id(), warps = blockDim.x >> 5;
    uint32_t best_n = 0, best_r = 0;
    uint32_t r = blockIdx.x * warps + (threadIdx.x >> 5), end = rows, step = gridDim.x * warps;
    if (segments != nullptr) {
        const SegmentTile t = segments[blockIdx.x];
        r = t.seg_start + t.first + (threadIdx.x >> 5);
        end = t.seg_start + min(t.first + kTile, t.seg_len);
        step = warps;
        tops += t.part;
        if constexpr (FORM == kRowsCentred) centre += (uint64_t) t.part * dim;
    }
    for (; r < end; r += step) {
        const float *row = data + (uint64_t) r * dim;
        float s = 0.0f, t = 0.0f;
        if constexpr (FORM == kRowsInPlace) {
            const float4 *row4 = reinterpret_cast<const float4 *>(row);   // dim % 4 == 0 and aligned, or a padded copy would be wanted
            for (uint32_t k = lane; k < (dim >> 2); k += 32) {
                const float4 v = __ldg(row4 + k);
                const float4 l = make_float4(tf32_rest(v.x), tf32_rest(v.y), tf32_rest(v.z), tf32_rest(v.w));
                s += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
                t += l.x * l.x + l.y * l.y + l.z * l.z + l.w * l.w;
            }
        } else {
            float *copy = padded + (uint64_t) (r - padded_from) * pitch;
            for (uint32_t k = lane; k < pitch; k += 32) {
                float v = k < dim ? __ldg(row + k) : 0.0f;
                if constexpr (FORM == kRowsCentred) v -= k < dim ? __ldg(centre + k) : 0.0f;
                const float l = tf32_rest(v);
                copy[k] = v;
                s += v * v;
                t += l * l;
            }
        }
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) {
            s += __shfl_xor_sync(kFullMask, s, off);
            t += __shfl_xor_sync(kFullMask, t, off);
        }
        const bool far = !(s < kFarNorm);
        if (lane == 0) {
            norms[r] = far ? __int_as_float(0x7f800000) : s;
            if (rest) rest[r] = far ? 0.0f : t;
        }
        best_n = max(best_n, far ? 0u : __float_as_uint(s));
        best_r = max(best_r, far ? 0u : __float_as_uint(t));
    }
    if (lane == 0) {
        atomicMax(&top[0], best_n);
        atomicMax(&top[1], best_r);
    }
    __syncthreads();
    if (tops && threadIdx.x == 0) {
        atomicMax(&tops->norm, top[0]);
        atomicMax(&tops->rest, top[1]);
    }
}

void (*rows_kernel(bool pad, bool centred))(const float *, uint32_t, uint32_t, float *, float *, uint32_t, float *, uint32_t, TruthTops *, const SegmentTile *,
                                            const float *) {
    return centred ? truth_rows_kernel<kRowsCentred> : (pad ? truth_rows_kernel<kRowsPadded> : truth_rows_kernel<kRowsInPlace>);
}

// 32 / fold minima, 16-byte aligned; m is FLT_MAX again afterwards.
__device__ __forceinline__ void store_minima(float (&m)[32], uint32_t fold, float *out) {
    if (fold >= 2u) {
#pragma unroll
        for (int j = 0; j < 16; j++) m[j] = fminf(m[j], m[j + 16]);
    }
    if (fold >= 4u) {
#pragma unroll
        for (int j = 0; j < 8; j++) m[j] = fminf(m[j], m[j + 8]);
    }
    if (fold >= 8u) {
#pragma unroll
        for (int j = 0; j < 4; j++) m[j] = fminf(m[j], m[j + 4]);
    }
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
        if (out != nullptr && (uint32_t) j < 32u / fold) *reinterpret_cast<float4 *>(out + j) = make_float4(m[j], m[j + 1], m[j + 2], m[j + 3]);
    }
#pragma unroll
    for (int j = 0; j < 32; j++) m[j] = FLT_MAX;
}

// Maps of the base rows: a call of one stride has one, partitions have strides of their own.
constexpr uint32_t kMaxStride = 16;
struct SampleMaps {
    CUtensorMap of[kMaxStride];              // by stride - 1
};
__device__ __forceinline__ const CUtensorMap *map_of(const CUtensorMap &m, uint32_t) { return &m; }
__device__ __forceinline__ const CUtensorMap *map_of(const SampleMaps &m, uint32_t stride) { return m.of + (stride - 1u); }

// SAMPLE: the sample pass, a kernel of its own for the registers of its minima (in one kernel the select pass took 4 % longer).
template<bool SAMPLE, typename Maps>
__global__ void __launch_bounds__(kTruthThreads) truth_umma_kernel(const TruthArgs a, const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ Maps tm_b) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *base = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t) 1023);
    const uint32_t kblocks = a.kblocks, stages = a.stages;
    const bool resident = kblocks <= kResidentBlocks;
    const uint32_t stage_bytes = resident ? kBlockBytes : 2 * kBlockBytes;   // a block of rows, then one of queries
    uint8_t *As = base, *ring = base + (resident ? kblocks * kBlockBytes : 0u);
    float *cn_w = reinterpret_cast<float *>(ring + stages * stage_bytes);     // a warp's column norms
    uint64_t *bars = reinterpret_cast<uint64_t *>(cn_w + kEpi * 32);
    uint64_t *a_full = bars, *full = bars + 1, *freed = full + stages, *mma_done = freed + stages, *tmem_free = mma_done + 2, *drained = tmem_free + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drained + 1);
    volatile uint32_t *failed = tmem_slot + 1;

    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bool seg = a.segments != nullptr;
    const SegmentTile part_of = seg ? a.segments[blockIdx.x] : SegmentTile{0, a.n, 0, a.stride, a.span, a.runs};
    const uint32_t qtiles = seg ? 1u : (a.Q + kTile - 1) / kTile;
    const uint32_t q0 = seg ? blockIdx.x * kTile : (blockIdx.x % qtiles) * kTile;      // index of the first query's results
    const uint32_t q_row = seg ? part_of.seg_start + part_of.first - a.map_from : q0;   // its row in the query map
    const uint32_t slice = seg ? 0u : blockIdx.x / qtiles, slices = seg ? 1u : a.slices;
    const uint32_t b_row = part_of.seg_start, m_row = b_row - a.map_from, stride = SAMPLE ? part_of.stride : 1u;
    const uint32_t n = part_of.seg_len / stride, all = (n + kTile - 1) / kTile;             // columns, tiles of them
    // a query of the CTA, by thread: one that wants candidates?
    bool wanted = tid < kTile && (seg ? part_of.first + tid < part_of.seg_len : q0 + tid < a.Q);
    if (wanted && !SAMPLE) wanted = __ldg(a.thr + q0 + tid) != -__int_as_float(0x7f800000);

    if (tid == 0) {
        mbar_init(a_full, 1);
        mbar_init(drained, 1);
        for (uint32_t s = 0; s < stages; s++) { mbar_init(full + s, 1); mbar_init(freed + s, 1); }
        for (int c = 0; c < 2; c++) { mbar_init(mma_done + c, 1); mbar_init(tmem_free + c, kEpi); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        *failed = a.give_up ? 1u : 0u;
    }
    if (warp == kEpi) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(2 * kTile) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    const bool any_wanted = __syncthreads_or(wanted);
    fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tiles = any_wanted && slice < all ? (all - slice + slices - 1) / slices : 0u;   // of this CTA

    uint32_t copies = 0;   // ring stages asked for, by the thread that copies
    if (warp == kEpi + 1) {
        // ================= copies: one thread =================
        if (lane == 0 && tiles > 0) {
            if (resident) {
                mbar_expect_tx(a_full, kblocks * kBlockBytes);
                for (uint32_t kb = 0; kb < kblocks; kb++) tma_load_2d(As + kb * kBlockBytes, &tm_q, kb * kBlock, q_row, a_full);
            }
            uint32_t s = 0, use = 0;
            bool ok = true;
            for (uint32_t t = 0; t < tiles && ok; t++) {
                const uint32_t c0 = (slice + t * slices) * kTile;
                for (uint32_t kb = 0; kb < kblocks; kb++) {
                    if (use > 0 && !mbar_wait(freed + s, (use - 1) & 1u, failed)) { ok = false; break; }
                    uint8_t *dst = ring + s * stage_bytes;
                    mbar_expect_tx(full + s, stage_bytes);
                    if constexpr (SAMPLE) tma_load_3d(dst, map_of(tm_b, stride), kb * kBlock, m_row % stride, m_row / stride + c0, full + s);
                    else tma_load_2d(dst, map_of(tm_b, 1u), kb * kBlock, m_row + c0, full + s);
                    if (!resident) tma_load_2d(dst + kBlockBytes, &tm_q, kb * kBlock, q_row, full + s);
                    copies++;
                    if (++s == stages) { s = 0; use++; }
                }
            }
        }
    } else if (warp == kEpi) {
        // ================= MMAs: one thread =================
        if (lane == 0 && tiles > 0) {
            const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((kTile >> 3) << 17) | ((kTile >> 4) << 24);
            const uint32_t a_addr = smem_u32(As), r_addr = smem_u32(ring);
            bool ok = !resident || mbar_wait(a_full, 0, failed);
            uint32_t s = 0, use = 0;
            for (uint32_t t = 0; t < tiles && ok; t++) {
                const uint32_t acc = t & 1u;
                if (t >= 2) ok = mbar_wait(tmem_free + acc, ((t >> 1) - 1) & 1u, failed);
                for (uint32_t kb = 0; kb < kblocks && ok; kb++) {
                    ok = mbar_wait(full + s, use & 1u, failed);
                    if (!ok) break;
                    fence_after();
                    const uint32_t b = r_addr + s * stage_bytes, q = resident ? a_addr + kb * kBlockBytes : b + kBlockBytes;
#pragma unroll
                    for (uint32_t k = 0; k < kBlock / 8; k++)
                        mma_tf32(tmem_base + acc * kTile, desc_sw128(q + k * 32u), desc_sw128(b + k * 32u), idesc, kb + k > 0 ? 1u : 0u);
                    commit_to(freed + s);
                    if (++s == stages) { s = 0; use++; }
                }
                if (ok) commit_to(mma_done + acc);
            }
        }
    } else {
        // ================= epilogue: thread (query, part) owns 32 columns of every tile =================
        const uint32_t quad = warp & 3u, part = warp >> 2, q = q0 + quad * 32u + lane;
        bool active = seg ? part_of.first + quad * 32u + lane < part_of.seg_len : q < a.Q;
        const float thr = (active && !SAMPLE) ? __ldg(a.thr + q) : 0.0f;
        active = active && thr != -__int_as_float(0x7f800000);
        float *cn = cn_w + warp * 32u;
        auto norm_of = [&](uint32_t t) {
            const uint32_t c = (slice + t * slices) * kTile + part * 32u + lane;
            return t < tiles && c < n ? __ldg(a.norms + b_row + c * stride) : 0.0f;
        };
        float ahead = norm_of(0);
        float m[32];
#pragma unroll
        for (int j = 0; j < 32; j++) m[j] = FLT_MAX;
        uint32_t run = 0, left = part_of.span;
        float *minima = active ? a.gmin + (uint64_t) q * a.groups + (slice * part_of.runs * kTile + part * 32u) / a.fold : nullptr;
        for (uint32_t t = 0; t < tiles; t++) {
            __syncwarp();
            cn[lane] = ahead;
            ahead = norm_of(t + 1);
            __syncwarp();
            const uint32_t acc = t & 1u, c0 = (slice + t * slices) * kTile + part * 32u;
            bool ok = !*failed && mbar_wait(mma_done + acc, (t >> 1) & 1u, failed);
            ok = __all_sync(kFullMask, ok);
            if (!ok) break;
            fence_after();
            uint32_t r[32];
            tmem_load32(tmem_base + ((quad * 32u) << 16) + acc * kTile + part * 32u, r);
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tmem_free + acc);
            float e[32];
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
                const float4 c4 = *reinterpret_cast<const float4 *>(cn + j);
                e[j] = __fmaf_rn(-2.0f, __uint_as_float(r[j]), c4.x);
                e[j + 1] = __fmaf_rn(-2.0f, __uint_as_float(r[j + 1]), c4.y);
                e[j + 2] = __fmaf_rn(-2.0f, __uint_as_float(r[j + 2]), c4.z);
                e[j + 3] = __fmaf_rn(-2.0f, __uint_as_float(r[j + 3]), c4.w);
            }
            if (c0 + 32u > n) {
#pragma unroll
                for (int j = 0; j < 32; j++)
                    if (c0 + j >= n) e[j] = FLT_MAX;
            }
            if (SAMPLE) {
#pragma unroll
                for (int j = 0; j < 32; j++) m[j] = fminf(m[j], e[j]);
                if (--left == 0 || t + 1 == tiles) {
                    store_minima(m, a.fold, minima ? minima + run * (kTile / a.fold) : nullptr);
                    run++;
                    left = part_of.span;
                }
            } else if (active) {
                float least = e[0];
#pragma unroll
                for (int j = 1; j < 32; j++) least = fminf(least, e[j]);
                if (least <= thr) {   // rare
#pragma unroll
                    for (int j = 0; j < 32; j++) {
                        if (e[j] <= thr && c0 + j < n) {
                            const uint32_t at = atomicAdd(a.count + q, 1u);
                            if (at < a.cap) a.cand[(uint64_t) q * a.cap + at] = c0 + j;
                        }
                    }
                }
            }
        }
        if (SAMPLE)   // spans that this CTA has no tile for
            for (; run < part_of.runs; run++) store_minima(m, a.fold, minima ? minima + run * (kTile / a.fold) : nullptr);
        if (*failed && lane == 0) atomicExch(a.gave_up, 1u);
    }
    fence_before();
    __syncthreads();
    if (*failed) {   // otherwise the epilogue has seen the last MMA, and that all copies
        if (warp == kEpi + 1 && lane == 0 && tiles > 0) {
            if (resident) mbar_drain(a_full, 0);
            drain_copies(full, stages, copies);
        }
        if (warp == kEpi && lane == 0) drain_mmas(drained);
        __syncthreads();
    }
    if (warp == kEpi) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2 * kTile) : "memory");
}

__device__ __forceinline__ uint32_t ordered(float x) {   // ascending floats as ascending integers
    const uint32_t u = __float_as_uint(x);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float from_ordered(uint32_t o) { return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o); }

// A CTA per query: the k-th smallest of its group minima (or, on later base passes, its k-th result so far) plus the error
// bounds. Also clears the query's candidate counter. Where the sample says that far more rows than `cap` will meet the
// threshold (`n` rows in all, `cols` of them sampled), the query is handed back before the pass over all tiles.
__global__ void __launch_bounds__(128) truth_threshold_kernel(const float *__restrict__ gmin, uint32_t groups, uint32_t k, const u64 *__restrict__ best,
                                                              const float *__restrict__ q_norm, const float *__restrict__ q_rest, uint32_t dim,
                                                              const SegmentTile *segments, const TruthTops *tops, uint32_t n, uint32_t cols, uint32_t cap,
                                                              const TruthBad bad, float *thr, uint32_t *count) {
    extern __shared__ uint32_t keys[];   // a thread reads those that it has written itself
    __shared__ uint32_t part[2][4];
    const uint32_t q = blockIdx.x, tid = threadIdx.x;
    __shared__ uint32_t range[4][3];     // by warp: smallest and largest key of the groups that have a row, their number
    // the CTA's sum; calls take turns with the two sets of words, so that one barrier each is enough
    uint32_t turn = 0;
    auto cta_sum = [&](uint32_t x) {
        x = __reduce_add_sync(kFullMask, x);
        if ((tid & 31u) == 0) part[turn][tid >> 5] = x;
        __syncthreads();
        x = part[turn][0] + part[turn][1] + part[turn][2] + part[turn][3];
        turn ^= 1u;
        return x;
    };
    auto keys_to = [&](uint32_t limit) {
        uint32_t c = 0;
        for (uint32_t i = tid; i < groups; i += 128) c += keys[i] <= limit ? 1u : 0u;
        return c;
    };
    uint32_t row = q, pitch = groups, item = q;   // the query's row in q_norm and q_rest, minima per query in gmin
    if (best != nullptr && thr[q] == -__int_as_float(0x7f800000)) return;   // handed back by an earlier pass
    if (segments != nullptr) {
        const SegmentTile t = segments[q / kTile];
        const uint32_t r = t.first + q % kTile;
        if (r >= t.seg_len) return;
        row = t.seg_start + r;
        groups = t.runs * kTile;
        k = min(k, t.seg_len);
        n = t.seg_len;
        cols = t.seg_len / t.stride;
        tops += t.part;
        item = 2u * t.index + (r - t.first) / (kTile / 2);
    }
    float kth;
    uint32_t with_row = 0;
    if (best == nullptr) {
        uint32_t lo = 0xffffffffu, hi = 0, has_row = 0;
        for (uint32_t i = tid; i < groups; i += 128) {
            const uint32_t key = ordered(gmin[(uint64_t) q * pitch + i]);
            keys[i] = key;
            if (key < ordered(FLT_MAX)) {
                lo = min(lo, key);
                hi = max(hi, key);
                has_row++;
            }
        }
        lo = __reduce_min_sync(kFullMask, lo);
        hi = __reduce_max_sync(kFullMask, hi);
        has_row = __reduce_add_sync(kFullMask, has_row);
        if ((tid & 31u) == 0) {
            range[tid >> 5][0] = lo;
            range[tid >> 5][1] = hi;
            range[tid >> 5][2] = has_row;
        }
        __syncthreads();
        lo = min(min(range[0][0], range[1][0]), min(range[2][0], range[3][0]));
        hi = max(max(range[0][1], range[1][1]), max(range[2][1], range[3][1]));
        with_row = range[0][2] + range[1][2] + range[2][2] + range[3][2];
        while (lo < hi) {   // the smallest key with at least k keys at or below it
            const uint32_t mid = lo + ((hi - lo) >> 1);
            if (cta_sum(keys_to(mid)) >= k) hi = mid; else lo = mid + 1;
        }
        kth = with_row >= k ? from_ordered(lo) : FLT_MAX;   // (beyond every bound: the query is handed back)
    } else {
        kth = __uint_as_float((uint32_t) (best[(uint64_t) q * k + k - 1] >> 32)) - q_norm[row];
    }
    const float qn = sqrtf(q_norm[row]), ql = sqrtf(q_rest[row]);
    const float bn = sqrtf(__uint_as_float(tops->norm)), bl = sqrtf(__uint_as_float(tops->rest));
    // |2 q.b - 2 tf32(q).tf32(b)| <= 2 (|q| |b - tf32(b)| + |q - tf32(q)| |b|); every sum (the two norms, the MMA's, the
    // fp32 distance) is within dim + 8 steps of 2^-23 of its terms' magnitudes, all below (|q| + |b|)^2
    const float sums = (float) (dim + 64u) * 4.0f * 1.1920929e-7f * (qn + bn) * (qn + bn);
    const float E = 1.001f * 2.0f * (qn * bl + ql * bn) + sums + 1e-30f;
    const float t = kth + 2.0f * E;
    bool good = fabsf(t) < kFarBound && q_norm[row] < kFarQuery;
    if (best == nullptr && n > cap) {
        // of G groups that have a row, g have one at or below t: (1 - p)^(cols / G) = 1 - g / G for the share p of such rows
        const float G = (float) with_row;
        auto expected = [&](float limit) {
            const float share = fminf((float) cta_sum(keys_to(ordered(limit))), G - 0.5f) / G;
            return (1.0f - expf(logf(1.0f - share) * G / (float) cols)) * (float) n;
        };
        if (expected(t) > 1.25f * (float) cap) {
            // were the bound nothing, the k-th smallest itself would be the threshold
            const bool hopeful = expected(kth) < 0.5f * (float) cap;
            if (tid == 0 && good && hopeful) atomicAdd(bad.hopeful, 1u);
            good = false;
        }
    }
    if (tid != 0) return;
    thr[q] = good ? t : -__int_as_float(0x7f800000);
    count[q] = 0;
    if (!good) report_bad(bad, item);
}

// Ascending dimensions, one fused multiply-add each: the order of bruteforce_tile_kernel and segment_knn_kernel.
__device__ __forceinline__ float direct_distance(const float *query, const float *__restrict__ row, uint32_t dim) {
    float acc = 0.0f;
    if ((dim & 3u) == 0 && (reinterpret_cast<uintptr_t>(row) & 15u) == 0) {
#pragma unroll 8
        for (uint32_t d = 0; d < dim; d += 4) {
            const float4 b = __ldg(reinterpret_cast<const float4 *>(row + d));
            const float4 x = *reinterpret_cast<const float4 *>(query + d);
            const float dx = x.x - b.x, dy = x.y - b.y, dz = x.z - b.z, dw = x.w - b.w;
            acc = __fmaf_rn(dx, dx, acc);
            acc = __fmaf_rn(dy, dy, acc);
            acc = __fmaf_rn(dz, dz, acc);
            acc = __fmaf_rn(dw, dw, acc);
        }
    } else {
#pragma unroll 8
        for (uint32_t d = 0; d < dim; d++) {
            const float df = query[d] - __ldg(row + d);
            acc = __fmaf_rn(df, df, acc);
        }
    }
    return acc;
}

// Sorts `total` keys in shared memory (room for the next power of two) by a CTA of 128 threads.
__device__ __forceinline__ void sort_keys(u64 *keys, uint32_t total) {
    const uint32_t tid = threadIdx.x;
    uint32_t size = 1;
    while (size < total) size <<= 1;
    for (uint32_t i = total + tid; i < size; i += 128) keys[i] = ~0ull;
    for (uint32_t span = 2; span <= size; span <<= 1)
        for (uint32_t step = span >> 1; step >= 1; step >>= 1) {
            __syncthreads();
            for (uint32_t p = tid; p < size / 2; p += 128) {
                const uint32_t i = 2 * (p & ~(step - 1u)) + (p & (step - 1u)), j = i + step;
                const u64 x = keys[i], y = keys[j];
                if ((x > y) == ((i & span) == 0)) { keys[i] = y; keys[j] = x; }
            }
        }
    __syncthreads();
}

// A CTA per query: exact distances of the candidates (and the earlier passes' results), sorted by (distance, id).
__global__ void __launch_bounds__(128) truth_rerank_kernel(const float *__restrict__ base, uint32_t first_row, const float *__restrict__ queries, uint32_t dim,
                                                           const uint32_t *__restrict__ cand, const uint32_t *__restrict__ count, uint32_t k, u64 *best,
                                                           bool earlier, int metric, uint32_t *out_ids, float *out_dists, float *thr, const TruthBad bad) {
    extern __shared__ __align__(16) uint32_t smem[];
    u64 *keys = reinterpret_cast<u64 *>(smem);                      // 4096
    float *query = reinterpret_cast<float *>(keys + 4096);          // dim
    const uint32_t q = blockIdx.x, tid = threadIdx.x;
    const uint32_t found = count[q], n = min(found, kCap);
    const uint32_t total = n + (earlier ? k : 0u);
    if (thr[q] == -__int_as_float(0x7f800000)) return;
    for (uint32_t d = tid; d < dim; d += 128) query[d] = queries[(uint64_t) q * dim + d];
    __syncthreads();
    if (found > kCap || total < k) {
        if (tid == 0) {
            thr[q] = -__int_as_float(0x7f800000);
            report_bad(bad, q);
        }
        return;
    }
    for (uint32_t i = tid; i < n; i += 128) {
        const uint32_t id = first_row + cand[(uint64_t) q * kCap + i];
        keys[i] = ((u64) __float_as_uint(direct_distance(query, base + (uint64_t) id * dim, dim)) << 32) | id;
    }
    if (earlier)
        for (uint32_t i = tid; i < k; i += 128) keys[n + i] = best[(uint64_t) q * k + i];
    sort_keys(keys, total);
    for (uint32_t i = tid; i < k && i < total; i += 128) {
        best[(uint64_t) q * k + i] = keys[i];
        if (out_ids) out_ids[(uint64_t) q * k + i] = (uint32_t) keys[i];
        if (out_dists) out_dists[(uint64_t) q * k + i] = finish_metric(__uint_as_float((uint32_t) (keys[i] >> 32)), metric);
    }
}

// Segment form, a CTA per row: its candidates without itself, nearest first, as partition-local ids; a row with fewer
// than out_degree others is padded with xorshift32(flat index) % partition size (nn_descent.cuh:1384-1391).
__global__ void __launch_bounds__(128) segment_rerank_kernel(const float *__restrict__ data, uint32_t dim, const SegmentTile *__restrict__ segments,
                                                             const uint32_t *__restrict__ cand, const uint32_t *__restrict__ count, uint32_t out_degree,
                                                             uint32_t row_base, int32_t *out, const float *__restrict__ thr, const TruthBad bad) {
    extern __shared__ __align__(16) uint32_t smem[];
    u64 *keys = reinterpret_cast<u64 *>(smem);                      // kSegCap
    float *query = reinterpret_cast<float *>(keys + kSegCap);       // dim
    const uint32_t q = blockIdx.x, tid = threadIdx.x;
    const SegmentTile t = segments[q / kTile];
    const uint32_t r = t.first + q % kTile;
    if (r >= t.seg_len) return;
    const float *seg = data + (uint64_t) t.seg_start * dim;
    const uint32_t found = count[q], n = min(found, kSegCap);
    const uint32_t want = min(out_degree, t.seg_len - 1u);
    if (thr[q] == -__int_as_float(0x7f800000)) return;
    if (found > kSegCap || n < want + 1u) {
        if (tid == 0) report_bad(bad, 2u * t.index + (r - t.first) / (kTile / 2));
        return;
    }
    for (uint32_t d = tid; d < dim; d += 128) query[d] = seg[(uint64_t) r * dim + d];
    __syncthreads();
    for (uint32_t i = tid; i < n; i += 128) {
        const uint32_t id = cand[(uint64_t) q * kSegCap + i];
        keys[i] = id == r ? ~0ull : ((u64) __float_as_uint(direct_distance(query, seg + (uint64_t) id * dim, dim)) << 32) | id;
    }
    sort_keys(keys, n);
    for (uint32_t j = tid; j < out_degree; j += 128) {
        const uint64_t flat = (uint64_t) (t.seg_start + r) * out_degree + j;
        uint32_t u = (uint32_t) (flat + (uint64_t) row_base * out_degree);  // xorshift32, utils.cuh:14-19
        u ^= u >> 13; u ^= u << 27; u ^= u >> 5; u *= 0x9E3779B9u;
        out[flat] = (int32_t) (j < want && j < n ? (uint32_t) keys[j] : u % t.seg_len);
    }
}

size_t up256(size_t x) { return (x + 255) & ~(size_t) 255; }

// The sample of a pass over n rows for k neighbours, taken by `slices` CTAs per query tile: every stride-th row. The
// select pass lets about stride x k columns through, the sample costs 1 / stride of it: 16 where at least 64 k rows remain,
// less for smaller sets. 8 k minima or more, so that few of the k smallest share one: a thread's 32 columns over as many tiles as
// that leaves; where few queries spread over many CTAs give 64 k and more, a thread folds its columns (every minimum costs the
// threshold kernel time; a fold of eight still keeps four neighbours in the file apart). At least min(k, n) minima have a row:
// with one tile all of its rows have a minimum each, with more the first one fills 128, or 32 k and more are left.
struct Sample {
    uint32_t stride, slices, span, runs, fold, groups;
};
Sample sample_of(uint32_t n, uint32_t k, uint32_t slices) {
    Sample s;
    s.stride = std::min(std::max(n / (64u * k), 1u), kMaxStride);
    const uint32_t tiles = (n / s.stride + kTile - 1) / kTile;
    s.slices = std::min(slices, tiles);
    const uint32_t per = (tiles + s.slices - 1) / s.slices;
    const uint32_t runs = std::min(per, (8u * k + kTile * s.slices - 1) / (kTile * s.slices));
    s.span = (per + runs - 1) / runs;
    s.runs = (per + s.span - 1) / s.span;
    s.fold = 1;
    while (s.fold < 8 && s.slices * s.runs * kTile / s.fold >= 64u * k) s.fold *= 2;
    s.groups = s.slices * s.runs * kTile / s.fold;
    return s;
}

uint32_t sm_count() {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 1;
    return (uint32_t) sms;
}

// CTAs per query tile of a pass: a full wave where the tiles suffice
uint32_t slices_of(uint32_t nq, uint32_t sms) { return std::max(1u, sms / ((nq + kTile - 1) / kTile)); }

struct TruthPlan {
    uint32_t nb, qb, pitch;     // rows and queries per pass, padded row length
    bool pad;
    Sample sample, sample_last;   // of a full pass over queries, of the last one
    size_t bad, items, tops, centre, norms, rows, q_rows, q_norm, q_rest, thr, count, cand, gmin, best, total;
};

TruthPlan truth_plan(const TcPasses &passes, const float *base, const float *queries, uint32_t n, uint32_t Q, uint32_t dim, uint32_t k, bool centred) {
    TruthPlan p;
    p.pad = centred || (dim & 3u) != 0 || ((reinterpret_cast<uintptr_t>(base) | reinterpret_cast<uintptr_t>(queries)) & 15u) != 0;
    p.pitch = (dim + 3u) & ~3u;
    p.nb = std::min(n, std::max(k, passes.base_rows));   // the first pass has k results
    if (p.pad && (uint64_t) p.nb * p.pitch > passes.padded_values) p.nb = std::max(k, passes.padded_values / p.pitch);
    p.qb = Q < passes.queries ? Q : passes.queries;
    const uint32_t last = Q % p.qb ? Q % p.qb : p.qb, sms = sm_count();
    p.sample = sample_of(p.nb, k, slices_of(p.qb, sms));
    p.sample_last = sample_of(p.nb, k, slices_of(last, sms));
    size_t at = 0;
    auto take = [&](size_t bytes) { const size_t o = at; at += up256(bytes); return o; };
    p.items = take((size_t) Q * 4);   // first: what it lists is answered from the rest of the scratch
    p.bad = take(sizeof(TcLeft) + sizeof(TruthTops));
    p.tops = p.bad + sizeof(TcLeft);
    p.centre = take(centred ? (size_t) dim * 4 : 0);
    p.norms = take((size_t) p.nb * 4);
    p.q_norm = take((size_t) p.qb * 4);
    p.q_rest = take((size_t) p.qb * 4);
    p.thr = take((size_t) p.qb * 4);
    p.count = take((size_t) p.qb * 4);
    p.cand = take((size_t) p.qb * kCap * 4);
    p.gmin = take(std::max((size_t) p.qb * p.sample.groups, (size_t) last * p.sample_last.groups) * 4);
    p.best = take((size_t) p.qb * k * 8);
    p.rows = take(p.pad ? (size_t) p.nb * p.pitch * 4 : 0);
    p.q_rows = take(p.pad ? (size_t) p.qb * p.pitch * 4 : 0);
    p.total = at;
    return p;
}

uint32_t ring_stages(uint32_t kblocks) { return kblocks <= kResidentBlocks ? 12u - kblocks : 6u; }    // 192 KB of operand blocks
size_t umma_smem(uint32_t stages) { return 1024 + 12u * (size_t) kBlockBytes + kEpi * 32 * 4 + (1 + 2 * stages + 5) * 8 + 16; }

// row-major rows of `pitch` floats as TMA boxes of 32 values x 128 rows (make_row_map takes the row length as the pitch)
bool row_map(CUtensorMap *tm, const float *ptr, uint32_t rows, uint32_t pitch) { return make_row_map(tm, ptr, rows, pitch, kTile); }

}  // namespace

// A kernel is loaded when its attributes are first asked for; most builds whose rows knn_tc.cu does not take come here.
cudaError_t preload_truth_kernels() {
    cudaFuncAttributes f;
    const void *kernels[] = {reinterpret_cast<const void *>(truth_rows_kernel<kRowsInPlace>), reinterpret_cast<const void *>(truth_rows_kernel<kRowsPadded>),
                             reinterpret_cast<const void *>(truth_umma_kernel<false, CUtensorMap>),
                             reinterpret_cast<const void *>(truth_umma_kernel<true, CUtensorMap>),
                             reinterpret_cast<const void *>(truth_umma_kernel<true, SampleMaps>),
                             reinterpret_cast<const void *>(truth_threshold_kernel), reinterpret_cast<const void *>(truth_rerank_kernel),
                             reinterpret_cast<const void *>(segment_rerank_kernel)};
    for (const void *k : kernels) {
        const cudaError_t e = cudaFuncGetAttributes(&f, k);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// Below 2^20 products of values a dozen launches cost what the tiles do (the smallest size timed is 1.3 x 2^20: 122 to 71 us).
bool truth_tc_eligible(uint32_t n, uint32_t Q, uint32_t dim, uint32_t k) {
    return dim >= 16 && dim <= 4096 && k >= 1 && k <= 128 && n >= 1 && (uint64_t) n * Q * dim >= (1ull << 20) && encode_tiled_fn() != nullptr;
}

size_t truth_tc_scratch_bytes(const TcPasses &passes, const float *base, const float *queries, uint32_t n, uint32_t Q, uint32_t dim, uint32_t k, bool centred) {
    return truth_plan(passes, base, queries, n, Q, dim, k, centred).total;
}

// What is left for the caller to answer by other means: see TcLeft. Synchronises the stream.
cudaError_t launch_truth_tc(const TcPasses &passes, const float *base, uint32_t n, const float *queries, uint32_t Q, uint32_t dim, uint32_t k, int metric,
                            bool centred, void *scratch, uint32_t *out_ids, float *out_dists, TcLeft *h_left, cudaStream_t stream) {
    const TruthPlan p = truth_plan(passes, base, queries, n, Q, dim, k, centred);
    char *w = static_cast<char *>(scratch);
    auto at = [&](size_t o) { return reinterpret_cast<float *>(w + o); };
    TcLeft *left = reinterpret_cast<TcLeft *>(w + p.bad);
    TruthTops *tops = reinterpret_cast<TruthTops *>(w + p.tops);
    TruthBad bad{&left->everything, &left->items, reinterpret_cast<uint32_t *>(w + p.items), &left->hopeful, nullptr, 0};
    float *centre = centred ? at(p.centre) : nullptr;
    float *norms = at(p.norms), *q_norm = at(p.q_norm), *q_rest = at(p.q_rest), *thr = at(p.thr), *gmin = at(p.gmin);
    uint32_t *count = reinterpret_cast<uint32_t *>(w + p.count), *cand = reinterpret_cast<uint32_t *>(w + p.cand);
    u64 *best = reinterpret_cast<u64 *>(w + p.best);
    *h_left = TcLeft{1, 0, 0};
    const uint32_t sms = sm_count();
    cudaError_t e = cudaMemsetAsync(left, 0, sizeof(TcLeft) + sizeof(TruthTops), stream);
    if (e != cudaSuccess) return e;
    if (centred) truth_centre_kernel<<<(dim + 127) / 128, 128, 0, stream>>>(base, n, dim, nullptr, centre);

    TruthArgs a{};
    a.dim = dim; a.cap = kCap; a.give_up = passes.give_up; a.kblocks = (p.pitch + kBlock - 1) / kBlock;
    a.stages = ring_stages(a.kblocks);
    a.norms = norms; a.thr = thr; a.gmin = gmin; a.count = count; a.cand = cand; a.gave_up = bad.gave_up;
    const size_t smem = umma_smem(a.stages);
    if ((e = cudaFuncSetAttribute(truth_umma_kernel<true, CUtensorMap>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(truth_umma_kernel<false, CUtensorMap>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem)) != cudaSuccess) return e;
    const size_t rr_smem = 4096 * 8 + (size_t) p.pitch * 4;
    if (rr_smem > 48 * 1024 && (e = cudaFuncSetAttribute(truth_rerank_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) rr_smem)) != cudaSuccess) return e;

    for (uint32_t qa = 0; qa < Q; qa += p.qb) {
        const uint32_t nq = Q - qa < p.qb ? Q - qa : p.qb;
        const float *qrows = queries + (size_t) qa * dim;
        float *q_padded = p.pad ? at(p.q_rows) : nullptr;
        rows_kernel(p.pad, centred)<<<(nq + 7) / 8, 256, 0, stream>>>(qrows, nq, dim, q_norm, q_rest, p.pitch, q_padded, 0, nullptr, nullptr, centre);
        bad.first = qa;
        CUtensorMap tm_q, tm_b;
        CUtensorMap tm_s;   // every stride-th row
        if (!row_map(&tm_q, p.pad ? q_padded : qrows, nq, p.pitch)) return cudaSuccess;
        a.Q = nq;
        const uint32_t qtiles = (nq + kTile - 1) / kTile;
        for (uint32_t ba = 0; ba < n; ba += p.nb) {
            const uint32_t nr = n - ba < p.nb ? n - ba : p.nb;
            const float *brows = base + (size_t) ba * dim;
            float *b_padded = p.pad ? at(p.rows) : nullptr;
            const uint32_t blocks = std::min((nr + 7) / 8, 8u * sms);
            rows_kernel(p.pad, centred)<<<blocks, 256, 0, stream>>>(brows, nr, dim, norms, nullptr, p.pitch, b_padded, 0, tops, nullptr, centre);
            if (!row_map(&tm_b, p.pad ? b_padded : brows, nr, p.pitch)) return cudaSuccess;
            a.n = nr;
            if (ba == 0) {
                const Sample &m = nq == p.qb ? p.sample : p.sample_last;
                if (!make_strided_row_map(&tm_s, p.pad ? b_padded : brows, nr, p.pitch, m.stride, kTile)) return cudaSuccess;
                a.slices = m.slices;
                a.stride = m.stride; a.span = m.span; a.runs = m.runs; a.fold = m.fold; a.groups = m.groups;
                truth_umma_kernel<true, CUtensorMap><<<qtiles * m.slices, kTruthThreads, smem, stream>>>(a, tm_q, tm_s);
                truth_threshold_kernel<<<nq, 128, (size_t) m.groups * 4, stream>>>(gmin, m.groups, k, nullptr, q_norm, q_rest, dim, nullptr, tops, nr, nr / m.stride, kCap,
                                                                                       bad, thr, count);
            } else {
                truth_threshold_kernel<<<nq, 128, 0, stream>>>(nullptr, 0, k, best, q_norm, q_rest, dim, nullptr, tops, nr, 0, kCap, bad, thr, count);
            }
            a.slices = std::min(slices_of(nq, sms), (nr + kTile - 1) / kTile);
            truth_umma_kernel<false, CUtensorMap><<<qtiles * a.slices, kTruthThreads, smem, stream>>>(a, tm_q, tm_b);
            const bool last = ba + nr == n;
            truth_rerank_kernel<<<nq, 128, rr_smem, stream>>>(base, ba, qrows, dim, cand, count, k, best, ba > 0, metric,
                                                              last ? out_ids + (size_t) qa * k : nullptr, last && out_dists ? out_dists + (size_t) qa * k : nullptr, thr, bad);
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
        }
    }
    if ((e = cudaMemcpyAsync(h_left, left, sizeof(TcLeft), cudaMemcpyDeviceToHost, stream)) != cudaSuccess) return e;
    return cudaStreamSynchronize(stream);
}

// ---- every row's nearest rows of its own partition ----------------------------------------------
namespace {

// Rows that TMA cannot read are copied, padded, a run of whole partitions at a time.
struct SegChunk {
    uint32_t row, rows, tile, tiles;   // its rows; its tiles in the call's table
};

std::vector<SegChunk> seg_chunks(const TcPasses &passes, bool pad, uint32_t pitch, uint32_t rows, const uint32_t *h_start, const uint32_t *h_len, uint32_t S,
                                 uint32_t max_len) {
    std::vector<SegChunk> chunks;
    uint32_t tile = 0;
    for (uint32_t s = 0; s < S; s++) {
        if (h_len[s] == 0 || h_len[s] > max_len) continue;
        const uint32_t tiles = (h_len[s] + kTile - 1) / kTile, end = h_start[s] + h_len[s];
        if (chunks.empty() || (pad && (uint64_t) (end - chunks.back().row) * pitch > passes.padded_values)) chunks.push_back({pad ? h_start[s] : 0u, 0, tile, 0});
        chunks.back().rows = pad ? end - chunks.back().row : rows;
        chunks.back().tiles += tiles;
        tile += tiles;
    }
    return chunks;
}

struct SegPlan {
    bool pad;
    uint32_t pitch, groups;
    std::vector<SegChunk> chunks;
    size_t bad, items, seen, tops, centre, tiles, norms, rest, thr, count, cand, gmin, rows, total;
};

SegPlan seg_plan(const TcPasses &passes, const float *data, uint32_t rows, uint32_t dim, const uint32_t *h_start, const uint32_t *h_len, uint32_t S, uint32_t max_len, uint32_t out_degree,
                 bool centred) {
    SegPlan p;
    p.pad = centred || (dim & 3u) != 0 || (reinterpret_cast<uintptr_t>(data) & 15u) != 0;
    p.pitch = (dim + 3u) & ~3u;
    p.groups = 1;
    size_t tiles = 0, parts = 0;
    for (uint32_t s = 0; s < S; s++)
        if (h_len[s] > 0 && h_len[s] <= max_len) {
            parts++;
            const uint32_t g = sample_of(h_len[s], out_degree + 1, 1).groups;
            if (g > p.groups) p.groups = g;
            tiles += (h_len[s] + kTile - 1) / kTile;
        }
    const size_t slots = (size_t) (tiles < passes.tiles ? tiles : passes.tiles) * kTile;
    size_t at = 0;
    auto take = [&](size_t bytes) { const size_t o = at; at += up256(bytes); return o; };
    p.bad = take(sizeof(TcLeft) + 2 * tiles * 4 + parts * sizeof(TruthTops));
    p.seen = p.bad + sizeof(TcLeft);
    p.tops = p.seen + 2 * tiles * 4;
    p.items = take(2 * tiles * 4);
    p.centre = take(centred ? parts * dim * 4 : 0);
    p.tiles = take(tiles * sizeof(SegmentTile));
    p.norms = take((size_t) rows * 4);
    p.rest = take((size_t) rows * 4);
    p.thr = take(slots * 4);
    p.count = take(slots * 4);
    p.cand = take(slots * kSegCap * 4);
    p.gmin = take(slots * p.groups * 4);
    p.chunks = seg_chunks(passes, p.pad, p.pitch, rows, h_start, h_len, S, max_len);
    uint32_t padded = 0;
    for (const SegChunk &c : p.chunks) padded = std::max(padded, c.rows);
    p.rows = take(p.pad ? (size_t) padded * p.pitch * 4 : 0);
    p.total = at;
    return p;
}

}  // namespace

// The padded copy of a partition that TMA cannot read is bounded, and so are its minima.
bool segment_tc_eligible(const float *data, uint32_t dim, const uint32_t *h_len, uint32_t S, uint32_t max_len, uint32_t out_degree) {
    const bool pad = (dim & 3u) != 0 || (reinterpret_cast<uintptr_t>(data) & 15u) != 0;
    if (dim < 16 || dim > 4096 || out_degree < 1 || out_degree > 64 || encode_tiled_fn() == nullptr) return false;
    uint64_t taken = 0, pairs = 0;
    for (uint32_t s = 0; s < S; s++) {
        if (h_len[s] > max_len) continue;
        if (h_len[s] > kSegRows || (pad && (uint64_t) h_len[s] * dim > (1ull << 30))) return false;
        taken += h_len[s];
        pairs += (uint64_t) h_len[s] * h_len[s];
    }
    // values a row meets: below 2^15 (about 1,000 rows of 32 values) the re-rank of a hundred candidates costs more than the pairs.
    // segment_knn_kernel against this, ms (uniform rows): 60 partitions of 1,000 x 23 0.97 / 1.41; 2 of 2,000 x 20 0.36 / 0.25; 8 of
    // 1,000 x 768 1.01 / 0.82; 4 of 15,000 x 50 9.8 / 7.2; 10 of 10,000 x 100 16.5 / 6.7, one of them with 3,000 equal rows 16.4 /
    // 9.0; 200 of 3,000 x 36 22.2 / 12.4; 15 of 4,000 x 960 (lists of 64) 34.1 / 17.0
    return pairs * dim >= taken << 15;
}

size_t segment_tc_scratch_bytes(const TcPasses &passes, const float *data, uint32_t rows, uint32_t dim, const uint32_t *h_start, const uint32_t *h_len, uint32_t S,
                                uint32_t max_len, uint32_t out_degree, bool centred) {
    return seg_plan(passes, data, rows, dim, h_start, h_len, S, max_len, out_degree, centred).total;
}

// Exact kNN rows of every partition of at most max_len rows: what segment_knn_kernel writes, bit for bit. What is left for that
// kernel: *h_all everything, otherwise h_tiles, three words each (its tiles). Synchronises the stream.
cudaError_t launch_segment_tc(const TcPasses &passes, const float *data, uint32_t rows, uint32_t dim, const uint32_t *h_start, const uint32_t *h_len,
                              uint32_t S, uint32_t max_len, uint32_t out_degree, uint32_t row_base, bool centred, void *scratch, int32_t *out, TcLeft *h_left,
                              std::vector<uint32_t> *h_tiles, cudaStream_t stream) {
    const SegPlan p = seg_plan(passes, data, rows, dim, h_start, h_len, S, max_len, out_degree, centred);
    std::vector<SegmentTile> tiles;
    uint32_t parts = 0;
    for (uint32_t s = 0; s < S; s++) {
        if (h_len[s] == 0 || h_len[s] > max_len) continue;
        const Sample m = sample_of(h_len[s], out_degree + 1, 1);
        for (uint32_t first = 0; first < h_len[s]; first += kTile) tiles.push_back(SegmentTile{h_start[s], h_len[s], first, m.stride, m.span, m.runs, parts, (uint32_t) tiles.size()});
        parts++;
    }
    h_tiles->clear();
    *h_left = TcLeft{0, 0, 0};
    if (tiles.empty()) return cudaSuccess;
    h_left->everything = 1;
    char *w = static_cast<char *>(scratch);
    auto at = [&](size_t o) { return reinterpret_cast<float *>(w + o); };
    TcLeft *left = reinterpret_cast<TcLeft *>(w + p.bad);
    TruthTops *tops = reinterpret_cast<TruthTops *>(w + p.tops);
    const TruthBad bad{&left->everything, &left->items, reinterpret_cast<uint32_t *>(w + p.items), &left->hopeful, reinterpret_cast<uint32_t *>(w + p.seen), 0};
    float *centre = centred ? at(p.centre) : nullptr;
    SegmentTile *d_tiles = reinterpret_cast<SegmentTile *>(w + p.tiles);
    uint32_t *count = reinterpret_cast<uint32_t *>(w + p.count), *cand = reinterpret_cast<uint32_t *>(w + p.cand);
    float *padded = p.pad ? at(p.rows) : nullptr;
    cudaError_t e = cudaMemsetAsync(left, 0, sizeof(TcLeft) + 2 * tiles.size() * 4 + parts * sizeof(TruthTops), stream);
    // the table is pageable host memory: the copy has read it when the call returns
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_tiles, tiles.data(), tiles.size() * sizeof(SegmentTile), cudaMemcpyHostToDevice, stream);
    if (e != cudaSuccess) return e;
    TruthArgs a{};
    a.dim = dim; a.cap = kSegCap; a.give_up = passes.give_up; a.kblocks = (p.pitch + kBlock - 1) / kBlock; a.stages = ring_stages(a.kblocks);
    a.groups = p.groups;
    a.fold = 1;
    a.norms = at(p.norms); a.thr = at(p.thr); a.gmin = at(p.gmin); a.count = count; a.cand = cand; a.gave_up = bad.gave_up;
    const size_t smem = umma_smem(a.stages), rr_smem = (size_t) kSegCap * 8 + (size_t) p.pitch * 4;
    if ((e = cudaFuncSetAttribute(truth_umma_kernel<true, SampleMaps>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(truth_umma_kernel<false, CUtensorMap>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem)) != cudaSuccess) return e;
    for (const SegChunk &c : p.chunks) {
        // (a grid's second dimension ends at 65,535)
        for (uint32_t t = 0; centred && t < c.tiles; t += 32768)
            truth_centre_kernel<<<dim3((dim + 127) / 128, std::min(c.tiles - t, 32768u)), 128, 0, stream>>>(data, 0, dim, d_tiles + c.tile + t, centre);
        rows_kernel(p.pad, centred)<<<c.tiles, 256, 0, stream>>>(data, rows, dim, at(p.norms), at(p.rest), p.pitch, padded, c.row, tops, d_tiles + c.tile, centre);
        const float *mapped_rows = p.pad ? padded : data;
        CUtensorMap tm;
        SampleMaps tm_s{};
        if (!row_map(&tm, mapped_rows, c.rows, p.pitch)) return cudaSuccess;
        uint32_t mapped = 0;   // a bit per stride
        for (uint32_t i = c.tile; i < c.tile + c.tiles; i++) {
            const uint32_t stride = tiles[i].stride;
            if (mapped & (1u << stride)) continue;
            mapped |= 1u << stride;
            if (!make_strided_row_map(&tm_s.of[stride - 1], mapped_rows, c.rows, p.pitch, stride, kTile)) return cudaSuccess;
        }
        a.map_from = c.row;
        for (uint32_t first = 0; first < c.tiles; first += passes.tiles) {
            const uint32_t n = std::min(c.tiles - first, passes.tiles);
            a.segments = d_tiles + c.tile + first;
            truth_umma_kernel<true, SampleMaps><<<n, kTruthThreads, smem, stream>>>(a, tm, tm_s);
            truth_threshold_kernel<<<n * kTile, 128, (size_t) p.groups * 4, stream>>>(a.gmin, p.groups, out_degree + 1, nullptr, a.norms, at(p.rest), dim,
                                                                                      a.segments, tops, 0, 0, kSegCap, bad, at(p.thr), count);
            truth_umma_kernel<false, CUtensorMap><<<n, kTruthThreads, smem, stream>>>(a, tm, tm);
            segment_rerank_kernel<<<n * kTile, 128, rr_smem, stream>>>(data, dim, a.segments, cand, count, out_degree, row_base, out, at(p.thr), bad);
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
        }
    }
    TcLeft got{1, 0, 0};
    if ((e = cudaMemcpyAsync(&got, left, sizeof got, cudaMemcpyDeviceToHost, stream)) != cudaSuccess) return e;
    if ((e = cudaStreamSynchronize(stream)) != cudaSuccess || got.everything) return e;
    *h_left = got;
    if (got.items == 0) return cudaSuccess;
    std::vector<uint32_t> items(got.items);
    if ((e = cudaMemcpyAsync(items.data(), bad.items, items.size() * 4, cudaMemcpyDeviceToHost, stream)) != cudaSuccess) return e;
    if ((e = cudaStreamSynchronize(stream)) != cudaSuccess) return e;
    for (const uint32_t i : items) {
        const SegmentTile &t = tiles[i / 2];
        h_tiles->insert(h_tiles->end(), {t.seg_start, t.seg_len, t.first + (i % 2) * (kTile / 2)});
    }
    return cudaSuccess;
}

}  // namespace glide
