// SeaLevelStage.percentileCut on the device (SeaLevelStage.kt:146-200, 579-651), bit-exact.
//
// The reference finds the height with the asked share of the planet's area below it: a 4096-bin
// histogram of cos(latitude) row weights brackets the answer, then the bracketing bin's cells are
// sorted by (height bits, index) and walked until the area below reaches the target. Both sums are
// sequential double sums in the reference, and the answer can flip on their last bit, so both are
// reproduced exactly:
//  - the histogram: per (row, bin) cell counts are exact integers, and each bin's sequential sum
//    over the rows in order is rebuilt by one warp, 32 rows at a time: inside one binade of the
//    running sum every addition adds a whole number of ulps, so a chunk is an integer prefix sum
//    (cg::warp_seq_sum, on the integer pipes); a row whose additions cross a binade or meet a tie is
//    taken alone by cg::seq_repeat_add, which takes `count` equal additions in closed form
//    (csrc/cg_fpemu.h);
//  - the bins' walk and the bracket's, whose cells are sorted on the device: sequential sums by one CTA,
//    inside binades as integer scans (cg_seqwalk.cuh).
// min, max, the bin of a cell and the land/relative split are elementwise or exact reductions.
#include <climits>
#include <cmath>
#include <vector>

#include "cg_common.cuh"
#include "cg_fpemu.h"
#include "cg_internal.h"
#include "cg_seqwalk.cuh"

namespace cg {

namespace {

constexpr int BINS = 4096;   // SeaLevelStage.HISTOGRAM_BINS

struct CutState {
    unsigned lo_key, hi_key;   // ordered float keys for atomicMin / atomicMax
    float lowest, highest, per;
    int degenerate;            // 1: the answer is `lowest` (flat field or nothing below)
    int bracket_bin;
    int count;                 // cells in the bracket bin
    double below_bracket;
    float todays;              // the percentile's height, before the lowstand
    int land_cells;
};

__device__ __forceinline__ unsigned ordered_key(float f) {
    unsigned b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float from_ordered_key(unsigned u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

// SeaLevelStage.sortableBits (SeaLevelStage.kt:648-651).
__device__ __forceinline__ int sortable_bits(float v) {
    int bits = __float_as_int(v);
    return bits < 0 ? (bits ^ 0x7FFFFFFF) : bits;
}

__device__ __forceinline__ int bin_of(float v, float lowest, float per) {
    float x = __fmul_rn(__fsub_rn(v, lowest), per);
    int b = (int)x;   // Float.toInt(): truncation
    return b < 0 ? 0 : (b > BINS - 1 ? BINS - 1 : b);
}

__global__ void k_cut_init(CutState* s) {
    s->lo_key = 0xFFFFFFFFu;
    s->hi_key = 0u;
    s->count = 0;
    s->land_cells = 0;
    s->degenerate = 0;
}

__global__ void __launch_bounds__(256) k_minmax(const float* __restrict__ h, size_t N, CutState* s) {
    unsigned lo = 0xFFFFFFFFu, hi = 0u;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x) {
        unsigned k = ordered_key(h[i]);
        lo = min(lo, k);
        hi = max(hi, k);
    }
    // One atomic a CTA: every warp's, on the two words, took 13 us of a 512 x 256 cut.
    __shared__ unsigned wlo[8], whi[8];
    lo = __reduce_min_sync(0xFFFFFFFFu, lo);
    hi = __reduce_max_sync(0xFFFFFFFFu, hi);
    if ((threadIdx.x & 31) == 0) {
        wlo[threadIdx.x >> 5] = lo;
        whi[threadIdx.x >> 5] = hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) {
            lo = min(lo, wlo[w]);
            hi = max(hi, whi[w]);
        }
        atomicMin(&s->lo_key, lo);
        atomicMax(&s->hi_key, hi);
    }
}

// The range and the bins' scale (SeaLevelStage.kt:590-600), from the extremes; degenerate: the answer is the lowest.
struct CutRange {
    float lowest, highest, per;
    int degenerate;
};
__device__ __forceinline__ CutRange cut_range(const CutState* s, double target) {
    CutRange r;
    r.lowest = from_ordered_key(s->lo_key);
    r.highest = from_ordered_key(s->hi_key);
    r.degenerate = __fsub_rn(r.highest, r.lowest) <= 0.0f || target <= 0.0;
    r.per = r.degenerate ? 0.0f : __fdiv_rn((float)(BINS - 1), __fsub_rn(r.highest, r.lowest));
    return r;
}

// One CTA per row: exact cell counts of every bin in that row.
__global__ void __launch_bounds__(512) k_row_counts(const float* __restrict__ h, int W, double target, CutState* s,
                                                    unsigned* __restrict__ counts) {
    __shared__ unsigned sh[BINS];
    const CutRange r = cut_range(s, target);
    if (blockIdx.x == 0 && threadIdx.x == 0) {   // kept for the kernels after this one
        s->lowest = r.lowest;
        s->highest = r.highest;
        s->per = r.per;
        s->degenerate = r.degenerate;
        if (r.degenerate) s->todays = r.lowest;
    }
    if (r.degenerate) return;
    const float lo = r.lowest, per = r.per;
    for (int b = threadIdx.x; b < BINS; b += blockDim.x) sh[b] = 0u;
    __syncthreads();
    const float* rowp = h + (size_t)blockIdx.x * W;
    for (int c = threadIdx.x; c < W; c += blockDim.x) atomicAdd(&sh[bin_of(rowp[c], lo, per)], 1u);
    __syncthreads();
    unsigned* out = counts + (size_t)blockIdx.x * BINS;
    for (int b = threadIdx.x; b < BINS; b += blockDim.x) out[b] = sh[b];
}

// One warp per bin: the reference's sequential sum `histogram[bin] += rowWeights[row]`, in cell
// order, replayed exactly, 32 rows at a time (cg::warp_seq_sum). The rows that hold none of the bin's
// cells (most rows of a small grid) are dropped first: the others queue up in order in shared memory.
__global__ void __launch_bounds__(256) k_bin_sums(const unsigned* __restrict__ counts, const double* __restrict__ w,
                                                  int H, const CutState* s, double* __restrict__ hist) {
    __shared__ int q_row[8][64];
    __shared__ unsigned q_cnt[8][64];
    const int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (b >= BINS || s->degenerate) return;
    double acc = 0.0, before;
    int queued = 0;
    unsigned next = lane < H ? counts[(size_t)lane * BINS + b] : 0u;
    for (int base = 0; base < H; base += 32) {
        const int r = base + lane;
        const unsigned c = next;
        next = r + 32 < H ? counts[(size_t)(r + 32) * BINS + b] : 0u;
        const unsigned rows = __ballot_sync(0xFFFFFFFFu, c != 0u);
        if (!rows) continue;
        if (c != 0u) {
            const int at = queued + __popc(rows & ((1u << lane) - 1u));
            q_row[warp][at] = r;
            q_cnt[warp][at] = c;
        }
        queued += __popc(rows);
        __syncwarp();
        if (queued >= 32) {
            acc = warp_seq_sum(acc, w[q_row[warp][lane]], (int64_t)q_cnt[warp][lane], &before);
            __syncwarp();
            if (lane < queued - 32) {
                q_row[warp][lane] = q_row[warp][32 + lane];
                q_cnt[warp][lane] = q_cnt[warp][32 + lane];
            }
            queued -= 32;
            __syncwarp();
        }
    }
    if (queued > 0)
        acc = warp_seq_sum(acc, lane < queued ? w[q_row[warp][lane]] : 0.0,
                           lane < queued ? (int64_t)q_cnt[warp][lane] : 0, &before);
    if (lane == 0) hist[b] = acc;
}

// SeaLevelStage.kt:614-622: the first bin that brings the weight below up to the target, the bins'
// sequential sum told apart by predicted binades and chained (one thread adding 4096 doubles in turn took
// 140 us, a CTA scan for every binade the sum grows through 70, this 25).
__global__ void __launch_bounds__(seqwalk::kSSThreads) k_bracket_bin(const double* __restrict__ hist, double target,
                                                                     CutState* s) {
    using namespace seqwalk;
    static_assert(BINS <= kSSBlock, "the histogram is one block of values");
    __shared__ CtaSum sh;
    if (s->degenerate) return;
    if (threadIdx.x == 0) {
        sh.s = 0.0;
        sh.hit = -1;
    }
    const SumIn<double> in{hist, nullptr, 0, BINS, nullptr, nullptr, 0.0, nullptr, 0};
    __syncthreads();
    cta_advance<true>(in, 0, BINS, sh, true, target);
    if (threadIdx.x == 0) {
        s->bracket_bin = sh.hit >= 0 ? sh.hit : BINS - 1;
        s->below_bracket = sh.hit >= 0 ? sh.below : sh.s;
    }
}

__global__ void k_bracket_collect(const float* __restrict__ h, size_t N, CutState* s, long long* __restrict__ keys) {
    if (s->degenerate) return;
    const unsigned FULL = 0xFFFFFFFFu;
    const float lo = s->lowest, per = s->per;
    const int bracket = s->bracket_bin;
    const int lane = threadIdx.x & 31;
    // Whole warps step together, so the bracket's cells of a warp take one atomic (the list's order
    // does not matter: it is sorted next).
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t base = (size_t)blockIdx.x * blockDim.x; base < N; base += stride) {
        const size_t i = base + threadIdx.x;
        const float v = i < N ? h[i] : 0.0f;
        const bool in = i < N && bin_of(v, lo, per) == bracket;
        const unsigned m = __ballot_sync(FULL, in);
        if (!m) continue;
        int slot = 0;
        if (lane == __ffs(m) - 1) slot = atomicAdd(&s->count, __popc(m));
        slot = __shfl_sync(FULL, slot, __ffs(m) - 1) + __popc(m & ((1u << lane) - 1u));
        if (in) keys[slot] = (long long)(((unsigned long long)(long long)sortable_bits(v) << 32) | (unsigned long long)i);
    }
}

// Up to SMALL_SORT keys sorted by rank, over the whole GPU: a warp takes RANK_KEYS keys, its lanes count
// the keys below each, and each goes to its count (the keys are distinct: they hold their cell). n^2 / 4
// loads and n^2 compares beat the n log^2 n of a bitonic network in one CTA, whose 66 steps of one CTA
// take 80 us at 2048 keys, up to 16384 keys; past that the network over chunks below is the faster.
constexpr int SMALL_SORT = 16384;
constexpr int RANK_KEYS = 4;
__global__ void __launch_bounds__(256) k_sort_rank(const long long* __restrict__ keys, const CutState* s,
                                                   long long* __restrict__ out) {
    const int n = s->count;
    if (s->degenerate || n > SMALL_SORT) return;
    const int lane = threadIdx.x & 31;
    const int k0 = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * RANK_KEYS;
    if (k0 >= n) return;
    long long mine[RANK_KEYS];
    int below[RANK_KEYS];
#pragma unroll
    for (int k = 0; k < RANK_KEYS; ++k) {
        mine[k] = k0 + k < n ? keys[k0 + k] : LLONG_MIN;
        below[k] = 0;
    }
    for (int i = lane; i < n; i += 32) {
        const long long other = keys[i];
#pragma unroll
        for (int k = 0; k < RANK_KEYS; ++k) below[k] += other < mine[k] ? 1 : 0;
    }
#pragma unroll
    for (int k = 0; k < RANK_KEYS; ++k) {
        const int rank = __reduce_add_sync(0xFFFFFFFFu, below[k]);
        if (lane == 0 && k0 + k < n) out[rank] = mine[k];
    }
}

// One compare-exchange stage of a global bitonic sort over P2 slots, padded with the largest key.
__global__ void k_sort_stage(long long* keys, int P2, int k, int j) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < P2; i += gridDim.x * blockDim.x) {
        int l = i ^ j;
        if (l <= i) continue;
        long long a = keys[i], b = keys[l];
        bool up = (i & k) == 0;
        if ((a > b) == up) {
            keys[i] = b;
            keys[l] = a;
        }
    }
}

// The bitonic network over P2 keys with its short strides in shared memory: a CTA holds a chunk of
// SORT_CH keys and takes every compare-exchange whose stride is below SORT_CH (directions from the
// keys' global positions, as in k_sort_stage); only the longer strides go through global memory,
// one launch each.
constexpr int SORT_CH = 4096;

__device__ __forceinline__ void chunk_steps(long long* sk, int base, int k, int jmax) {
    for (int j = jmax; j > 0; j >>= 1) {
        for (int p = threadIdx.x; p < SORT_CH / 2; p += blockDim.x) {
            const int i = (p & (j - 1)) | ((p & ~(j - 1)) << 1);
            const int l = i | j;
            const bool up = ((base + i) & k) == 0;
            const long long a = sk[i], b = sk[l];
            if ((a > b) == up) {
                sk[i] = b;
                sk[l] = a;
            }
        }
        __syncthreads();
    }
}

// Every stage k <= SORT_CH, whole, per chunk (merge = 0); or the strides below SORT_CH of stage k.
__global__ void __launch_bounds__(1024) k_sort_chunk(long long* keys, int merge) {
    __shared__ long long sk[SORT_CH];
    const int base = blockIdx.x * SORT_CH;
    for (int i = threadIdx.x; i < SORT_CH; i += blockDim.x) sk[i] = keys[base + i];
    __syncthreads();
    if (merge == 0) {
        for (int k = 2; k <= SORT_CH; k <<= 1) chunk_steps(sk, base, k, k >> 1);
    } else {
        chunk_steps(sk, base, merge, SORT_CH / 2);
    }
    for (int i = threadIdx.x; i < SORT_CH; i += blockDim.x) keys[base + i] = sk[i];
}

__global__ void k_pad(long long* keys, int n, int P2) {
    for (int i = n + blockIdx.x * blockDim.x + threadIdx.x; i < P2; i += gridDim.x * blockDim.x) keys[i] = LLONG_MAX;
}

// SeaLevelStage.kt:636-644: walk the sorted bracket until the area below reaches the target: the answer is the
// first cell whose sum before it does, so the one after the cell that brings the sum there. The sum is
// sequential; the CTA takes it 8192 cells at a time, inside binades as integer scans (cg_seqwalk.cuh). Scans
// with one warp replaying the rest of the chunk from the first crossing took 32 us at 2048 x 1024 and 455 at
// 8192 x 4096, this 9 and 90.
__global__ void __launch_bounds__(seqwalk::kSSThreads) k_bracket_walk(const float* __restrict__ h,
                                                                      const long long* __restrict__ keys,
                                                                      const double* __restrict__ w, int W, double target,
                                                                      int most, CutState* s, double* __restrict__ weights) {
    using namespace seqwalk;
    __shared__ CtaSum sh;
    if (s->degenerate) return;
    const int n = s->count;
    if (n > most) return;   // its keys are not sorted yet
    if (n == 0) {
        if (threadIdx.x == 0) s->todays = s->highest;
        return;
    }
    if (threadIdx.x == 0) {
        sh.s = s->below_bracket;
        sh.hit = -1;
    }
    for (int i = threadIdx.x; i < n; i += kSSThreads) weights[i] = w[pdiv((int)(keys[i] & 0xFFFFFFFFLL), W)];
    __syncthreads();
    int answer = s->below_bracket >= target ? 0 : n;
    const SumIn<double> in{weights, nullptr, 0, (size_t)n, nullptr, nullptr, 0.0, nullptr, 0};
    for (int base = 0; base < n && answer == n; base += kSSBlock) {
        cta_advance<true>(in, (size_t)base, min(n - base, kSSBlock), sh, false, target);
        __syncthreads();
        if (sh.hit >= 0) answer = base + sh.hit + 1;
        __syncthreads();
        if (answer != n) break;
    }
    if (threadIdx.x == 0) s->todays = h[(int)(keys[min(answer, n - 1)] & 0xFFFFFFFFLL)];
}

// SeaLevelStage.landAndWaterAt (SeaLevelStage.kt:175-200).
__global__ void k_land_and_water(const float* __restrict__ h, size_t N, int most, CutState* s, float lowstand,
                                 float land_half, float sea_half, uint8_t* __restrict__ land,
                                 float* __restrict__ rel) {
    if (!s->degenerate && s->count > most) return;   // the shoreline is not known yet
    const float shore = __fsub_rn(s->todays, lowstand);
    int count = 0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x) {
        float g = h[i];
        float d = __fsub_rn(g, shore);
        if (g >= shore) {
            land[i] = 1;
            rel[i] = __fdiv_rn(d, land_half);
            ++count;
        } else {
            land[i] = 0;
            rel[i] = __fdiv_rn(d, sea_half);
        }
    }
    for (int o = 16; o > 0; o >>= 1) count += __shfl_xor_sync(0xFFFFFFFFu, count, o);
    if ((threadIdx.x & 31) == 0 && count) atomicAdd(&s->land_cells, count);
}

}  // namespace

cg_status row_weights_dev(cg_ctx* ctx, int W, int H, const double** d_weights, double* total) {
    CG_BUF(double, d_w, ctx, S_ROWW, H);
    if (ctx->rw_w != W || ctx->rw_h != H) {
        // shorelineForFraction (SeaLevelStage.kt:580-584): a per-grid constant table, built once.
        std::vector<double> w(H);
        const double PI = 3.141592653589793;
        for (int row = 0; row < H; ++row) w[row] = std::cos(PI / 2 - (row + 0.5) / H * PI);
        double t = 0.0;
        for (int row = 0; row < H; ++row) t += w[row] * W;
        CG_CUDA(ctx, cudaMemcpyAsync(d_w, w.data(), sizeof(double) * H, cudaMemcpyHostToDevice, ctx->stream));
        CG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        ctx->rw_w = W;
        ctx->rw_h = H;
        ctx->rw_total = t;
    }
    *d_weights = d_w;
    *total = ctx->rw_total;
    return CG_OK;
}

cg_status percentile_cut_dev(cg_ctx* ctx, int W, int H, const float* d_h, float sea_level, float land_half,
                             float sea_half, float lowstand_share, uint8_t* d_land, float* d_rel, float* h_shoreline,
                             int* h_land_cells) {
    size_t N = (size_t)W * H;
    const double* d_w;
    double total;
    cg_status st = row_weights_dev(ctx, W, H, &d_w, &total);
    if (st != CG_OK) return st;
    float submerged = sea_level < 0.0f ? 0.0f : (sea_level > 1.0f ? 1.0f : sea_level);
    double target = (double)submerged * total;
    CG_BUF(CutState, d_s, ctx, S_SMALL, 1);
    CG_BUF(unsigned, d_counts, ctx, S_HIST, (size_t)H * BINS);
    CG_BUF(double, d_hist, ctx, S_SCRATCH4, BINS);
    CG_BUF(long long, d_keys, ctx, S_BRACKET, N);
    CG_BUF(double, d_weights, ctx, S_BRACKETW, N);   // the bracket's row weights
    cudaStream_t sm = ctx->stream;
    int grid = ctx->num_sms * 8;
    CG_LAUNCH(ctx) k_cut_init<<<1, 1, 0, sm>>>(d_s);
    CG_LAUNCH(ctx) k_minmax<<<grid, 256, 0, sm>>>(d_h, N, d_s);
    CG_LAUNCH(ctx) k_row_counts<<<H, 512, 0, sm>>>(d_h, W, target, d_s, d_counts);
    CG_LAUNCH(ctx) k_bin_sums<<<BINS * 32 / 256, 256, 0, sm>>>(d_counts, d_w, H, d_s, d_hist);
    CG_LAUNCH(ctx) k_bracket_bin<<<1, seqwalk::kSSThreads, 0, sm>>>(d_hist, target, d_s);
    CG_LAUNCH(ctx) k_bracket_collect<<<grid, 256, 0, sm>>>(d_h, N, d_s, d_keys);
    CG_CHECK_LAUNCH(ctx);
    // A bracket of up to SMALL_SORT cells, as nearly every one is, is sorted and walked before the host has
    // read its size; a larger one is left as it is by those launches, and sorted and walked after.
    CG_BUF(long long, d_sorted, ctx, S_BRACKET2, SMALL_SORT);
    CG_LAUNCH(ctx) k_sort_rank<<<SMALL_SORT / RANK_KEYS / 8, 256, 0, sm>>>(d_keys, d_s, d_sorted);
    auto walk = [&](const long long* keys, int most) {
        CG_LAUNCH(ctx) k_bracket_walk<<<1, seqwalk::kSSThreads, 0, sm>>>(d_h, keys, d_w, W, target, most, d_s, d_weights);
        CG_LAUNCH(ctx) k_land_and_water<<<grid, 256, 0, sm>>>(d_h, N, most, d_s, lowstand_share, land_half, sea_half,
                                                              d_land, d_rel);
    };
    walk(d_sorted, SMALL_SORT);
    CG_CHECK_LAUNCH(ctx);
    CutState hs;
    CG_TRY_ST(read_back(ctx, {{&hs, d_s, sizeof(hs)}}));
    if (!hs.degenerate && hs.count > SMALL_SORT) {
        int P2 = 1;
        while (P2 < hs.count) P2 <<= 1;
        int blocks = (P2 / 2 + 255) / 256;
        if (blocks > grid) blocks = grid;
        CG_LAUNCH(ctx) k_pad<<<blocks, 256, 0, sm>>>(d_keys, hs.count, P2);
        // P2 > SMALL_SORT >= SORT_CH: whole chunks of SORT_CH keys.
        CG_LAUNCH(ctx) k_sort_chunk<<<P2 / SORT_CH, 1024, 0, sm>>>(d_keys, 0);
        for (int k = 2 * SORT_CH; k <= P2; k <<= 1) {
            for (int j = k >> 1; j >= SORT_CH; j >>= 1)
                CG_LAUNCH(ctx) k_sort_stage<<<blocks, 256, 0, sm>>>(d_keys, P2, k, j);
            CG_LAUNCH(ctx) k_sort_chunk<<<P2 / SORT_CH, 1024, 0, sm>>>(d_keys, k);
        }
        walk(d_keys, INT_MAX);
        CG_CHECK_LAUNCH(ctx);
        CG_TRY_ST(read_back(ctx, {{&hs, d_s, sizeof(hs)}}));
    }
    *h_shoreline = hs.todays - lowstand_share;
    *h_land_cells = hs.land_cells;
    return CG_OK;
}

}  // namespace cg
