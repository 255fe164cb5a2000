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
// A block of 8192 values is taken by one CTA, 8 values a thread (cta_advance): a scan for the binade the
// sum is in, and the first value whose partial m leaves that binade found over the CTA. A block with such a
// crossing is told apart (cta_classify): a scan of the values in fixed point says which binade every
// partial sum is in, all but those next to a power of two; the values between two binades, and the few in
// doubt, are listed, and the chain adds those in hardware, one after another, and the runs of steps between
// them as integers. On GB300 a dependent chain of double additions fed from shared memory takes about 80 ns
// an addition, so a piece of 1024 taken one by one cost 80 us, and a CTA scan for every crossing 3 to 5.
//
// Sums of up to kDirectBlocks blocks run so from the first value, one CTA per sum. Longer ones tell their
// blocks apart in parallel first, each after an estimate of the sum before it, with a bound of how far that
// may be off. One warp then chains the blocks, those without a listed value 32 at a time, and a block that
// was not told apart, or whose steps do not apply, is taken by cta_advance. At 2048 x 1024 the flexure's load takes
// 0.18 ms (2.3 with a CTA scan for every crossing), a mean of rain 49 us (166).
#include <climits>
#include <cstdint>

#include "cg_common.cuh"
#include "cg_internal.h"
#include "cg_seqwalk.cuh"

namespace cg {
namespace {

using namespace seqwalk;

constexpr int kMaxSums = 5;                      // sums of one launch
// Sums up to this many blocks are taken by one CTA from the first value: a block costs about 6 us so, the
// parallel form's three launches about 20 us and little for more blocks.
constexpr int kDirectBlocks = 3;

// The sums of one launch.
template <typename T>
struct SumJobs {
    SumIn<T> in[kMaxSums];
};

// A block told apart (cta_classify) after the sum the blocks before it are estimated at: how many values are
// listed (-1: it was not), the binade of the first run of steps, the steps of all its runs, what its first run
// takes more from an odd sum, and the pieces of 1024 that hold a listed value; and a listed value, the steps of the block before it and the binade of the
// run after it.
struct BlockSteps {
    long long steps;
    int spec, listed, odd;
    unsigned pieces;
};
constexpr int kListed = kMostAlone;   // a block's listed values, at most; a block with more is taken by hand
struct Listed {
    long long steps;
    double value;
    int spec;
};

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

// A block's sum and the sum of its magnitudes, and how far those may be off: where its neighbours' sums
// begin, and how surely. In fixed point, in units of 2^-60 of what they can reach, on the integer pipes
// (double additions held the FP64 pipe for 12 us a launch).
struct Estimate {
    double sum, magnitude, off;
};
template <typename T>
__global__ void __launch_bounds__(kSSThreads) k_ss_estimate(SumJobs<T> jobs, Estimate* __restrict__ est) {
    __shared__ long long sums[kSSThreads / 32], spans[kSSThreads / 32];
    __shared__ int tops[kSSThreads / 32];
    const unsigned FULL = 0xFFFFFFFFu;
    const SumIn<T>& in = jobs.in[blockIdx.y];
    const size_t base = (size_t)blockIdx.x * kSSBlock;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (base >= in.n) return;
    T v[kSSPer];
    const unsigned has = load_values(in, base, v);
    int top = -1;
#pragma unroll
    for (int t = 0; t < kSSPer; ++t)
        if ((has >> t) & 1u) top = max(top, field_of(v[t]));
    top = __reduce_max_sync(FULL, top);
    if (lane == 0) tops[warp] = top;
    __syncthreads();
    top = __reduce_max_sync(FULL, tops[lane]);
    const int unit = max(top, 1) - kTopField<T> / 2 + 14 - 59;
    long long sum = 0, span = 0;
    if (top < kTopField<T>) {
#pragma unroll
        for (int t = 0; t < kSSPer; ++t) {
            const long long q = (has >> t) & 1u ? units_of(magnitude_of(v[t]), unit) : 0;
            sum += q;
            span += q < 0 ? -q : q;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        sum += __shfl_down_sync(FULL, sum, o);
        span += __shfl_down_sync(FULL, span, o);
    }
    if (lane == 0) {
        sums[warp] = sum;
        spans[warp] = span;
    }
    __syncthreads();
    if (warp == 0) {
        sum = sums[lane];
        span = spans[lane];
        for (int o = 16; o > 0; o >>= 1) {
            sum += __shfl_down_sync(FULL, sum, o);
            span += __shfl_down_sync(FULL, span, o);
        }
        if (lane == 0) {
            Estimate e{0.0, 0.0, 0.0};
            if (top == kTopField<T>) e.off = __longlong_as_double(0x7FF0000000000000LL);
            else if (top >= 0)
                e = Estimate{scalbn((double)sum, unit), scalbn((double)(span + kSSBlock), unit), scalbn((double)kSSBlock, unit)};
            est[in.first_block + blockIdx.x] = e;
        }
    }
}

// Each block told apart after the estimates before it. The rounded sum is off from the real sum by at most
// 2^-53 of the magnitudes before for every addition, n of them; adding up the estimates adds 64, and the
// estimates' own offs; all doubled for the magnitudes' own roundings.
template <typename T>
__global__ void __launch_bounds__(kSSThreads) k_ss_walks(SumJobs<T> jobs, const Estimate* __restrict__ est,
                                                        BlockSteps* __restrict__ blocks, Listed* __restrict__ lists) {
    __shared__ CtaSum sh;
    __shared__ Estimate part[kSSThreads / 32];
    __shared__ double2 start;
    const SumIn<T>& in = jobs.in[blockIdx.y];
    const size_t base = (size_t)blockIdx.x * kSSBlock;
    if (base >= in.n) return;
    Estimate s{0.0, 0.0, 0.0};
    auto over_warp = [&]() {
        for (int o = 16; o > 0; o >>= 1) {
            s.sum += __shfl_down_sync(0xFFFFFFFFu, s.sum, o);
            s.magnitude += __shfl_down_sync(0xFFFFFFFFu, s.magnitude, o);
            s.off += __shfl_down_sync(0xFFFFFFFFu, s.off, o);
        }
    };
    for (int i = (int)threadIdx.x; i < (int)blockIdx.x; i += kSSThreads) {
        const Estimate e = est[in.first_block + i];
        s.sum += e.sum;
        s.magnitude += e.magnitude;
        s.off += e.off;
    }
    if ((int)(threadIdx.x & ~31u) < (int)blockIdx.x) over_warp();   // the warps that hold an estimate
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        s = part[threadIdx.x];
        if (blockIdx.x > 32) over_warp();
        if (threadIdx.x == 0) {
            const double init = in.init ? *in.init : 0.0;
            start = make_double2(s.sum + init, ((double)base + 64.0) * 0x1p-52 * (s.magnitude + fabs(init)) + 2.0 * s.off);
        }
    }
    __syncthreads();
    const int len = (int)(in.n - base < (size_t)kSSBlock ? in.n - base : (size_t)kSSBlock);
    long long steps;
    int listed = cta_classify<false>(in, base, 0, len, start.x, start.y, kParityStart, sh, 0.0, &steps);
    if (listed > kListed) listed = -1;
    const int block = in.first_block + blockIdx.x;
    for (int k = threadIdx.x; k < listed; k += kSSThreads)
        lists[(size_t)block * kListed + k] = Listed{sh.steps[k], sh.values[k], sh.spec[k + 1]};
    if (threadIdx.x == 0) {
        unsigned pieces = 0;
        for (int k = 0; k < listed; ++k) pieces |= 1u << (sh.at[k] / kSSThreads);
        blocks[block] = BlockSteps{steps, sh.spec[0], listed, sh.odd, pieces};
    }
}

// s after a run of steps taken for the binade `spec` (-1: unchecked); false where they do not apply.
__device__ __forceinline__ bool take_steps(double& s, long long steps, int spec) {
    if (steps == 0) return true;
    const Binade b = binade_of(s);
    const long long m = b.m + steps;
    if (!b.normal || !inside(m) || (spec != -1 && spec != (b.ef | (b.neg << 11)))) return false;
    s = sum_of(b, m);
    return true;
}

// The chain over the blocks, one CTA a sum: warp 0 takes whole blocks without a listed value together, up to
// 32 by a scan, and the listed values of the others one by one (every lane the same); a block that was not
// told apart, or whose steps do not apply, is taken by the CTA.
template <typename T>
__global__ void __launch_bounds__(kSSThreads) k_ss_chain(SumJobs<T> jobs, const BlockSteps* __restrict__ heads,
                                                        const Listed* __restrict__ lists) {
    const unsigned FULL = 0xFFFFFFFFu;
    __shared__ CtaSum sh;
    __shared__ int sh_block;
    __shared__ Listed list[kListed];
    const SumIn<T>& in = jobs.in[blockIdx.x];
    const int blocks = (int)((in.n + kSSBlock - 1) / kSSBlock);
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0) sh.s = in.init ? *in.init : 0.0;
    __syncthreads();
    long long whole = 0, reduced = 0, alone = 0;
    auto count = [&](unsigned pieces) {
        const int a = __popc(pieces);
        whole += a == 0;
        reduced += a ? kSSPer - a : 0;
        alone += a;
    };
    for (int j = 0; j < blocks; ++j) {
        if (threadIdx.x < 32) {
            double s = sh.s;
            bool by_hand = false;
            while (j < blocks && !by_hand) {
                const int here = min(32, blocks - j);
                BlockSteps w{0, -1, 0, 0, 0};
                if (lane < here) w = heads[in.first_block + j + lane];
                int i = 0;
                while (i < here && !by_hand) {
                    // The blocks from i without a listed value, in the binade the sum is in.
                    const Binade b = binade_of(s);
                    const bool plain = w.listed == 0 && (w.spec < 0 ? w.steps == 0 : b.normal && w.spec == (b.ef | (b.neg << 11)));
                    Run run = run_identity();
                    if (lane >= i && plain) {
                        run.step[0] = w.steps;
                        run.step[1] = w.steps + w.odd;
                        run.out = (unsigned)(run.step[0] & 1) | ((unsigned)(1 + run.step[1]) & 1u) << 1;
                    }
                    const bool odd = __any_sync(FULL, plain && w.odd != 0);
                    const Run incl = warp_scan(run, odd);
                    const long long x = odd && (b.m & 1) ? incl.step[1] : incl.step[0];
                    const bool ok = plain && (w.spec < 0 || inside(wrap_add(b.m, x)));
                    const unsigned stop = __ballot_sync(FULL, !ok || lane >= here) & ~((1u << i) - 1u);
                    const int end = stop ? __ffs(stop) - 1 : 32;
                    if (end > i) {
                        const long long steps = __shfl_sync(FULL, x, end - 1);
                        if (b.normal) s = sum_of(b, wrap_add(b.m, steps));
                        whole += end - i;
                        i = end;
                        continue;
                    }
                    // Block i alone.
                    const int listed = __shfl_sync(FULL, w.listed, i);
                    long long all = __shfl_sync(FULL, w.steps, i);
                    const int more = b.normal && (b.m & 1) ? __shfl_sync(FULL, w.odd, i) : 0;
                    int spec = __shfl_sync(FULL, w.spec, i);
                    const unsigned pieces = __shfl_sync(FULL, w.pieces, i);
                    by_hand = listed <= 0;
                    if (by_hand) break;
                    for (int k = lane; k < listed; k += 32) list[k] = lists[(size_t)(in.first_block + j + i) * kListed + k];
                    __syncwarp();
                    double t = s;
                    long long done = 0;
                    bool sound = true;
                    for (int k = 0; k < listed; ++k) {
                        const Listed e = list[k];
                        sound &= take_steps(t, wrap_add(e.steps, (k == 0 ? more : 0) - done), spec);
                        t = __dadd_rn(t, e.value);
                        done = e.steps;
                        spec = e.spec;
                    }
                    sound &= take_steps(t, wrap_add(all, -done), spec);
                    __syncwarp();
                    by_hand = !sound;
                    if (by_hand) break;
                    s = t;
                    count(pieces);
                    ++i;
                }
                j += i;
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
        cta_advance(in, base, (int)(in.n - base < (size_t)kSSBlock ? in.n - base : (size_t)kSSBlock), sh, true);
        if (threadIdx.x == 0) count(sh.alone);
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
    CG_BUF(Estimate, d_est, ctx, S_SS_EST, (size_t)total);
    CG_BUF(BlockSteps, d_heads, ctx, S_SS_WALK, (size_t)total);
    CG_BUF(Listed, d_lists, ctx, S_SS_SPEC, (size_t)total * kListed);
    const dim3 grid(most, count);
    CG_LAUNCH(ctx) k_ss_estimate<T><<<grid, kSSThreads, 0, sm>>>(jobs, d_est);
    CG_LAUNCH(ctx) k_ss_walks<T><<<grid, kSSThreads, 0, sm>>>(jobs, d_est, d_heads, d_lists);
    CG_LAUNCH(ctx) k_ss_chain<T><<<count, kSSThreads, 0, sm>>>(jobs, d_heads, d_lists);
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
