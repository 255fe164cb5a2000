// The reference's sequential double sums of float fields (`var s = 0.0; for (c in cells) s += f[c]`:
// the rain and cover means of normaliseOverLand / shieldingOverLand, HydraulicErosion.kt:476-486,
// 557-567, and the flexure's load mean, Isostasy.kt:337-339) and of double terms (the belts' books),
// bit for bit, without a serial chain of double additions.
//
// Each addition rounds, so the sum depends on the order. But while the running sum s stays inside one
// binade [2^e, 2^(e+1)) (one sign), s is m u with m an integer in [2^52, 2^53) and u = 2^(e-52), and
// fl(s + x) = (m + r) u where r is x / u rounded to an integer, to nearest, ties to even: the tie's
// choice depends on the parity of m and nothing else, and a tie always leaves m even. So a run of
// additions inside a binade is an integer walk whose only state is m's parity, and a run's walks
// compose: a prefix scan over the values gives every partial m at once.
//
// A block of 8192 values is taken by one CTA, 8 values a thread (cta_advance): a scan for the binade
// the sum is in, the first value whose partial m leaves that binade found over the CTA, and that one
// addition taken in hardware; crossings cluster (a sum near zero changes sign many times), so one warp
// then goes on 32 values at a time until a window holds no crossing, and the CTA scans again from
// there. On GB300 a dependent chain of double additions fed from shared memory takes about 80 ns an
// addition, so a piece of 1024 taken one by one cost 80 us; a crossing costs one CTA scan, about 3 us.
// With the pieces taken one by one the 2048 x 1024 flexure took 13.5 ms a call, with the scans 5.1; the
// belts' replay at 1024 x 512 (five sums a round, each its own launches) 161 ms, and 79 with the scans
// and the five sums side by side.
//
// Sums of up to kDirectBlocks blocks run so from the first value, one CTA per sum. Longer ones reduce
// their blocks in parallel first, each under the binade an estimate of the running sum gives it: a
// block's reduction is, for each entering parity, its total step, its lowest and highest partial steps
// (which say whether the walk stays inside the binade) and its leaving parity. One warp then chains
// the reductions 32 at a time by a scan, and a block that is not in the binade it was reduced for, or
// does not stay in it, is taken by cta_advance.
#include <climits>
#include <cstdint>

#include "cg_common.cuh"
#include "cg_internal.h"
#include "cg_seqwalk.cuh"

namespace cg {
namespace {

using namespace seqwalk;

constexpr long long kBig = 1LL << 58;            // a partial step this large leaves any binade: give up
constexpr int kMaxSums = 5;                      // sums of one launch
// Sums up to this many blocks are taken by one CTA from the first value. A block taken so costs about
// 2.5 us, the parallel form's three launches about 25 us before its first block.
constexpr int kDirectBlocks = 10;

// The sums of one launch.
template <typename T>
struct SumJobs {
    SumIn<T> in[kMaxSums];
};

// A run of additions inside one binade, for each parity of m entering it.
struct Walk {
    long long step[2], lo[2], hi[2];   // total step; lowest and highest partial step (lo > hi: no values)
    int out[2];                        // parity of m leaving
    int fail;                          // a value the integer walk cannot hold (it leaves the binade)
    int spec;                          // the binade and sign it was made for (exponent | sign << 11), -1: none
    int zero;                          // no value adds anything
};

__device__ __forceinline__ Walk walk_identity() {
    Walk w;
    for (int q = 0; q < 2; ++q) {
        w.step[q] = 0;
        w.lo[q] = kBig;
        w.hi[q] = -kBig;
        w.out[q] = q;
    }
    w.fail = 0;
    w.spec = -1;
    w.zero = 1;
    return w;
}

// a then b.
__device__ __forceinline__ Walk walk_then(const Walk& a, const Walk& b) {
    Walk w;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const bool odd = a.out[q] != 0;
        const long long step = odd ? b.step[1] : b.step[0], lo = odd ? b.lo[1] : b.lo[0], hi = odd ? b.hi[1] : b.hi[0];
        w.step[q] = a.step[q] + step;
        const long long blo = a.step[q] + lo, bhi = a.step[q] + hi;
        w.lo[q] = lo > hi ? a.lo[q] : (a.lo[q] < blo ? a.lo[q] : blo);
        w.hi[q] = lo > hi ? a.hi[q] : (a.hi[q] > bhi ? a.hi[q] : bhi);
        w.out[q] = odd ? b.out[1] : b.out[0];
    }
    w.fail = a.fail | b.fail;
    w.zero = a.zero & b.zero;
    w.spec = a.spec;
    if (w.step[0] > kBig || w.step[0] < -kBig || w.step[1] > kBig || w.step[1] < -kBig) w.fail = 1;
    return w;
}

// The walk of a run of values in order, for both entering parities.
struct LocalWalk {
    Walk w;
    __device__ void init() { w = walk_identity(); }
    __device__ void add(const Step& st) {
        if (st.fail) w.fail = 1;
        for (int q = 0; q < 2; ++q) {
            const int p = w.out[q];
            const long long r = st.tie ? st.r + ((p + (int)(st.r & 1)) & 1) : st.r;
            w.step[q] += r;
            if (w.step[q] < w.lo[q]) w.lo[q] = w.step[q];
            if (w.step[q] > w.hi[q]) w.hi[q] = w.step[q];
            w.out[q] = st.tie ? 0 : (p ^ (int)(r & 1));
            if (w.step[q] > kBig || w.step[q] < -kBig) w.fail = 1;
        }
    }
};

__device__ __forceinline__ Walk shfl_walk(const Walk& w, int from) {
    Walk o;
    for (int q = 0; q < 2; ++q) {
        o.step[q] = __shfl_sync(0xFFFFFFFFu, w.step[q], from);
        o.lo[q] = __shfl_sync(0xFFFFFFFFu, w.lo[q], from);
        o.hi[q] = __shfl_sync(0xFFFFFFFFu, w.hi[q], from);
        o.out[q] = __shfl_sync(0xFFFFFFFFu, w.out[q], from);
    }
    o.fail = __shfl_sync(0xFFFFFFFFu, w.fail, from);
    o.zero = __shfl_sync(0xFFFFFFFFu, w.zero, from);
    o.spec = -1;
    return o;
}

// The warp's walks composed in lane order; lane 0 gets the result.
__device__ __forceinline__ Walk warp_walk(Walk w) {
    const int lane = threadIdx.x & 31;
    for (int off = 1; off < 32; off <<= 1) {   // lane i takes lanes i .. i + 2 off - 1, a tree over the lanes
        const Walk o = shfl_walk(w, (lane + off) & 31);
        if ((lane & (2 * off - 1)) == 0 && lane + off < 32) w = walk_then(w, o);
    }
    return w;
}

// The CTA's threads' walks composed in thread order; every thread calls it, thread 0 gets the result.
__device__ Walk cta_walk(const Walk& mine, Walk* sh_warps) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const Walk w = warp_walk(mine);
    if (lane == 0) sh_warps[warp] = w;
    __syncthreads();
    Walk total = walk_identity();
    if (warp == 0) total = warp_walk(lane < (int)(blockDim.x >> 5) ? sh_warps[lane] : walk_identity());
    return total;
}

template <typename T>
__device__ __forceinline__ void finish_sum(const SumIn<T>& in, double s, long long whole, long long reduced,
                                           long long alone) {
    *in.out = in.divisor != 0.0 ? __ddiv_rn(s, in.divisor) : s;
    if (in.counts) {
        in.counts[0] = whole;
        in.counts[1] = reduced;
        in.counts[2] = alone;
    }
}

// Sums of few blocks, a CTA each, from the first value to the last.
template <typename T>
__global__ void __launch_bounds__(kSSThreads) k_ss_direct(SumJobs<T> jobs) {
    __shared__ CtaSum sh;
    const SumIn<T>& in = jobs.in[blockIdx.x];
    if (threadIdx.x == 0) sh.s = in.init ? *in.init : 0.0;
    __syncthreads();
    long long whole = 0, reduced = 0, alone = 0;
    for (size_t base = 0; base < in.n; base += kSSBlock) {
        cta_advance(in, base, (int)(in.n - base < (size_t)kSSBlock ? in.n - base : (size_t)kSSBlock), sh);
        if (threadIdx.x == 0) {
            const int a = __popc(sh.alone);
            whole += a == 0;
            reduced += a ? kSSPer - a : 0;
            alone += a;
        }
        __syncthreads();   // sh.alone is read before the next block clears it
    }
    if (threadIdx.x == 0) finish_sum(in, sh.s, whole, reduced, alone);
}

// A cheap estimate of each block's sum (any order): it only picks the binade each block is reduced for.
template <typename T>
__global__ void __launch_bounds__(kSSThreads) k_ss_estimate(SumJobs<T> jobs, double* __restrict__ est) {
    __shared__ double part[kSSThreads / 32];
    const SumIn<T>& in = jobs.in[blockIdx.y];
    const size_t base = (size_t)blockIdx.x * kSSBlock;
    if (base >= in.n) return;
    double s = 0.0;
    for (int t = 0; t < kSSPer; ++t) {
        T v;
        if (value_at(in, base + (size_t)t * kSSThreads + threadIdx.x, &v)) s += (double)v;
    }
    for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xFFFFFFFFu, s, off);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        double t = part[threadIdx.x];
        for (int off = 16; off > 0; off >>= 1) t += __shfl_down_sync(0xFFFFFFFFu, t, off);
        if (threadIdx.x == 0) est[in.first_block + blockIdx.x] = t;
    }
}

// Each block's walk under the binade it is expected to begin in, that of the estimates before it. A
// thread's values are consecutive.
template <typename T>
__global__ void __launch_bounds__(kSSThreads) k_ss_walks(SumJobs<T> jobs, const double* __restrict__ est,
                                                        Walk* __restrict__ walks) {
    __shared__ Walk sh_warps[kSSThreads / 32];
    __shared__ double part[kSSThreads / 32];
    __shared__ int s_spec;
    const SumIn<T>& in = jobs.in[blockIdx.y];
    const size_t base = (size_t)blockIdx.x * kSSBlock;
    if (base >= in.n) return;
    T v[kSSPer];
    const unsigned has = load_values(in, base, v);
    double s = threadIdx.x == 0 && in.init ? *in.init : 0.0;
    for (int i = (int)threadIdx.x; i < (int)blockIdx.x; i += kSSThreads) s += est[in.first_block + i];
    if ((int)(threadIdx.x & ~31u) < (int)blockIdx.x || threadIdx.x < 32)   // the warps that hold an estimate
        for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xFFFFFFFFu, s, off);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        double t = part[threadIdx.x];
        for (int off = 16; off > 0; off >>= 1) t += __shfl_down_sync(0xFFFFFFFFu, t, off);
        if (threadIdx.x == 0) {
            const Binade b = binade_of(t);
            s_spec = b.normal ? (b.ef | (b.neg << 11)) : -1;
        }
    }
    __syncthreads();
    const int sp = s_spec;
    LocalWalk lw;
    lw.init();
#pragma unroll
    for (int t = 0; t < kSSPer; ++t)
        if (has & (1u << t)) {
            lw.w.zero = 0;
            if (sp >= 0) lw.add(step_of(v[t], sp & 0x7FF, sp >> 11));
        }
    Walk total = cta_walk(lw.w, sh_warps);
    if (threadIdx.x == 0) {
        total.spec = sp;
        walks[in.first_block + blockIdx.x] = total;
    }
}

// The chain over the blocks, one CTA a sum: warp 0 takes whole blocks 32 at a time while their walks
// apply, the CTA takes the block where one does not.
template <typename T>
__global__ void __launch_bounds__(kSSThreads) k_ss_chain(SumJobs<T> jobs, const Walk* __restrict__ walks) {
    const unsigned FULL = 0xFFFFFFFFu;
    __shared__ CtaSum sh;
    __shared__ int sh_block;
    const SumIn<T>& in = jobs.in[blockIdx.x];
    const int blocks = (int)((in.n + kSSBlock - 1) / kSSBlock);
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0) sh.s = in.init ? *in.init : 0.0;
    __syncthreads();
    long long whole = 0, reduced = 0, alone = 0;
    for (int j = 0; j < blocks; ++j) {
        if (threadIdx.x < 32) {
            double s = sh.s;
            while (j < blocks) {
                const int k = j + lane;
                Walk w = walk_identity();
                if (k < blocks) w = walks[in.first_block + k];
                const Binade b = binade_of(s);
                const bool zero = k < blocks && w.zero;
                bool ok = zero || (k < blocks && b.normal && !w.fail && w.spec == (b.ef | (b.neg << 11)));
                Run mine = run_identity();
                if (ok && !zero) {
                    mine.step[0] = w.step[0];
                    mine.step[1] = w.step[1];
                    mine.out = (unsigned)w.out[0] | ((unsigned)w.out[1] << 1);
                }
                const Run incl = warp_scan(mine, true);
                Run excl;
                excl.step[0] = __shfl_up_sync(FULL, incl.step[0], 1);
                excl.step[1] = __shfl_up_sync(FULL, incl.step[1], 1);
                excl.out = __shfl_up_sync(FULL, incl.out, 1);
                if (lane == 0) excl = run_identity();
                const bool odd = b.m & 1;
                const long long m = wrap_add(b.m, odd ? excl.step[1] : excl.step[0]);
                const long long after = wrap_add(b.m, odd ? incl.step[1] : incl.step[0]);
                if (ok && !zero) {
                    const int p = (int)(m & 1);
                    ok = (p ? w.lo[1] > w.hi[1] : w.lo[0] > w.hi[0]) ||
                         (inside(wrap_add(m, p ? w.lo[1] : w.lo[0])) && inside(wrap_add(m, p ? w.hi[1] : w.hi[0])));
                }
                const unsigned bad = __ballot_sync(FULL, !ok);
                const int taken = bad ? __ffs(bad) - 1 : 32;
                if (taken > 0 && b.normal) s = sum_of(b, __shfl_sync(FULL, after, taken - 1));
                whole += taken;
                j += taken;
                if (bad) break;
            }
            if (lane == 0) {
                sh.s = s;
                sh_block = j;
            }
        }
        __syncthreads();
        j = sh_block;
        if (j >= blocks) break;
        const size_t base = (size_t)j * kSSBlock;
        cta_advance(in, base, (int)(in.n - base < (size_t)kSSBlock ? in.n - base : (size_t)kSSBlock), sh);
        if (threadIdx.x == 0) {
            const int a = __popc(sh.alone);
            whole += a == 0;
            reduced += a ? kSSPer - a : 0;
            alone += a;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) finish_sum(in, sh.s, whole, reduced, alone);
}

// `count` sums in one set of launches.
template <typename T>
cg_status seq_sums_run(cg_ctx* ctx, SumJobs<T>& jobs, int count) {
    cudaStream_t sm = ctx->stream;
    int most = 0, total = 0;
    for (int i = 0; i < count; ++i) {
        const int blocks = (int)((jobs.in[i].n + kSSBlock - 1) / kSSBlock);
        jobs.in[i].first_block = total;
        total += blocks;
        most = blocks > most ? blocks : most;
    }
    if (most <= kDirectBlocks) {
        CG_LAUNCH(ctx) k_ss_direct<T><<<count, kSSThreads, 0, sm>>>(jobs);
        CG_CHECK_LAUNCH(ctx);
        return CG_OK;
    }
    CG_BUF(double, d_est, ctx, S_SS_EST, (size_t)total);
    CG_BUF(Walk, d_walks, ctx, S_SS_WALK, (size_t)total);
    const dim3 grid(most, count);
    CG_LAUNCH(ctx) k_ss_estimate<T><<<grid, kSSThreads, 0, sm>>>(jobs, d_est);
    CG_LAUNCH(ctx) k_ss_walks<T><<<grid, kSSThreads, 0, sm>>>(jobs, d_est, d_walks);
    CG_LAUNCH(ctx) k_ss_chain<T><<<count, kSSThreads, 0, sm>>>(jobs, d_walks);
    CG_CHECK_LAUNCH(ctx);
    return CG_OK;
}

}  // namespace

// The reference's sequential double sum of (mode 0) x or (mode 1) 1 - 0.5 x over the cells of `mask`
// (every cell when null), in cell order, into *d_out on the device; divided by `divisor` when it is
// not 0 (the mean's one division, in double).
cg_status seq_sum_dev(cg_ctx* ctx, const float* d_x, const uint8_t* d_mask, int mode, size_t n, double divisor,
                      double* d_out, long long* d_counts) {
    SumJobs<float> jobs{};
    jobs.in[0] = SumIn<float>{d_x, d_mask, mode, n, nullptr, d_out, divisor, d_counts, 0};
    return seq_sums_run(ctx, jobs, 1);
}

// `s = 0.0; for (v in x) s += v` over n double terms, into *d_out on the device.
cg_status seq_sum_f64_dev(cg_ctx* ctx, const double* d_x, size_t n, double* d_out) {
    SumJobs<double> jobs{};
    jobs.in[0] = SumIn<double>{d_x, nullptr, 0, n, nullptr, d_out, 0.0, nullptr, 0};
    return seq_sums_run(ctx, jobs, 1);
}

// `for (v in x) *total += v` for each running total, side by side.
cg_status seq_totals_f64_dev(cg_ctx* ctx, const SeqTotal* totals, int count) {
    static_assert(kSeqTotals <= kMaxSums, "a launch holds every total");
    if (count < 1 || count > kSeqTotals) return fail(ctx, CG_BAD_ARG, "%d running totals", count);
    SumJobs<double> jobs{};
    for (int i = 0; i < count; ++i)
        jobs.in[i] = SumIn<double>{totals[i].x, nullptr, 0, totals[i].n, totals[i].total, totals[i].total, 0.0, nullptr, 0};
    return seq_sums_run(ctx, jobs, count);
}

}  // namespace cg

using namespace cg;

extern "C" cg_status cg_sequential_sum(cg_ctx* ctx, const float* x, const uint8_t* mask, int32_t mode, int64_t n,
                                       double* sum, int64_t* counts) {
    if (!ctx || !sum || n < 0 || (n > 0 && !x) || (mode != 0 && mode != 1)) return CG_BAD_ARG;
    CG_CUDA(ctx, cudaSetDevice(ctx->device));
    ctx->run.active = false;
    const size_t N = (size_t)n;
    CG_BUF(float, d_x, ctx, S_SS_X, N);
    CG_BUF(uint8_t, d_m, ctx, S_SS_MASK, mask ? N : 1);
    CG_BUF(double, d_out, ctx, S_SS_OUT, 4);   // the sum, then the three counts
    if (N) CG_CUDA(ctx, cudaMemcpyAsync(d_x, x, N * sizeof(float), cudaMemcpyHostToDevice, ctx->stream));
    if (N && mask) CG_CUDA(ctx, cudaMemcpyAsync(d_m, mask, N, cudaMemcpyHostToDevice, ctx->stream));
    long long* d_counts = (long long*)(d_out + 1);
    CG_TRY_ST(seq_sum_dev(ctx, d_x, mask ? d_m : nullptr, mode, N, 0.0, d_out, d_counts));
    CG_CUDA(ctx, cudaMemcpyAsync(sum, d_out, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    if (counts) CG_CUDA(ctx, cudaMemcpyAsync(counts, d_counts, 3 * sizeof(long long), cudaMemcpyDeviceToHost, ctx->stream));
    CG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return CG_OK;
}
