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

namespace cg {
namespace {

constexpr int kSSThreads = 1024;
constexpr int kSSPer = 8;                        // values per thread in the parallel reduction
constexpr int kSSBlock = kSSThreads * kSSPer;    // values per block
constexpr long long kM0 = 1LL << 52, kM1 = 1LL << 53;
constexpr long long kBig = 1LL << 58;            // a partial step this large leaves any binade: give up
constexpr int kMaxSums = 5;                      // sums of one launch
// Sums up to this many blocks are taken by one CTA from the first value. A block taken so costs about
// 2.5 us, the parallel form's three launches about 25 us before its first block.
constexpr int kDirectBlocks = 10;

// The values summed: float fields (widened exactly), or double terms already in summation order.
template <typename T>
struct SumIn {
    const T* x;
    const uint8_t* mask;   // may be null: every value (float fields only)
    int mode;              // 0: x, 1: 1 - 0.5 x (the cover's shielding factor; float fields only)
    size_t n;
    const double* init;    // the sum before the first value (may be null: +0)
    double* out;           // may be `init`
    double divisor;        // the sum is divided by it unless it is 0
    long long* counts;     // may be null: how the sum went (3)
    int first_block;       // this sum's first entry in the launch's estimates and walks
};

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
    int zero;                          // every value is a zero: the block leaves any sum but -0 as it was
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

__device__ __forceinline__ bool value_at(const SumIn<float>& in, size_t i, float* v) {
    if (i >= in.n) return false;
    if (in.mask && !in.mask[i]) return false;
    const float x = in.x[i];
    *v = in.mode == 1 ? __fsub_rn(1.0f, __fmul_rn(0.5f, x)) : x;
    return true;
}

__device__ __forceinline__ bool value_at(const SumIn<double>& in, size_t i, double* v) {
    if (i >= in.n) return false;
    *v = in.x[i];
    return true;
}

// One value's step in the binade with exponent field ef (u = 2^(ef - 1075)), for a sum of sign `neg`:
// the step r when it is not a tie, else the tie's floor f (r = f + ((parity + f) & 1)). An absent value
// (a masked cell) adds nothing, as the reference skips it; +0 and -0 add nothing to a nonzero sum.
struct Step {
    long long r;
    int tie, fail;
};

__device__ __forceinline__ Step step_of(float v, int ef, int neg) {
    Step s{0, 0, 0};
    const uint32_t b = __float_as_uint(v);
    const int fe = (int)((b >> 23) & 0xFF);
    if (fe == 0xFF) {
        s.fail = 1;
        return s;
    }
    long long M = (long long)(b & 0x7FFFFF);
    if (fe != 0) M |= 1LL << 23;
    if (M == 0) return s;
    const bool negative = ((b >> 31) != 0) != (neg != 0);   // y's sign: x's, flipped for a negative sum
    // y = M 2^k with k = (max(fe, 1) - 150) - (ef - 1075)
    const int k = (fe == 0 ? 1 : fe) - 150 - ef + 1075;
    if (k >= 0) {
        if (k > 29) {
            s.fail = 1;
            return s;
        }
        s.r = negative ? -(M << k) : (M << k);
        return s;
    }
    const int sh = -k;
    if (sh >= 40) return s;   // |y| < 2^-16: rounds to 0
    const long long a = M >> sh, frac = M & ((1LL << sh) - 1), half = 1LL << (sh - 1);
    if (frac == half) {
        s.tie = 1;
        s.r = negative ? -(a + 1) : a;   // floor(y)
    } else {
        const long long r = a + (frac > half ? 1 : 0);
        s.r = negative ? -r : r;
    }
    return s;
}

// The same for a double value: y = M 2^k with M < 2^53 and k = max(fe, 1) - ef. A value of 2^58 u or
// more, or NaN or infinity, is left to the serial additions; below u / 4 it adds nothing.
__device__ __forceinline__ Step step_of(double v, int ef, int neg) {
    Step s{0, 0, 0};
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const int fe = (int)((b >> 52) & 0x7FF);
    if (fe == 0x7FF) {
        s.fail = 1;
        return s;
    }
    long long M = (long long)(b & ((1ULL << 52) - 1));
    if (fe != 0) M |= 1LL << 52;
    if (M == 0) return s;
    const bool negative = ((b >> 63) != 0) != (neg != 0);
    const int k = (fe == 0 ? 1 : fe) - ef;
    if (k >= 0) {
        if (k > 5) {
            s.fail = 1;
            return s;
        }
        s.r = negative ? -(M << k) : (M << k);
        return s;
    }
    const int sh = -k;
    if (sh >= 55) return s;   // |y| < 2^-2: rounds to 0
    const long long a = M >> sh, frac = M & ((1LL << sh) - 1), half = 1LL << (sh - 1);
    if (frac == half) {
        s.tie = 1;
        s.r = negative ? -(a + 1) : a;
    } else {
        const long long r = a + (frac > half ? 1 : 0);
        s.r = negative ? -r : r;
    }
    return s;
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

// A run's step and leaving parity for each entering parity (bit q of `out`: the parity left from q).
struct Run {
    long long step[2];
    unsigned out;
};
__device__ __forceinline__ long long wrap_add(long long a, long long b) {   // past a crossing the sums are not read
    return (long long)((unsigned long long)a + (unsigned long long)b);
}
__device__ __forceinline__ Run run_then(const Run& a, const Run& b) {
    Run r;
    const unsigned p0 = a.out & 1u, p1 = (a.out >> 1) & 1u;
    r.step[0] = wrap_add(a.step[0], p0 ? b.step[1] : b.step[0]);
    r.step[1] = wrap_add(a.step[1], p1 ? b.step[1] : b.step[0]);
    r.out = ((b.out >> p0) & 1u) | (((b.out >> p1) & 1u) << 1);
    return r;
}
// The inclusive scan of the warp's runs. Without ties both parities step alike: one sum does.
__device__ __forceinline__ Run warp_scan(Run r, bool ties) {
    const int lane = threadIdx.x & 31;
    for (int o = 1; o < 32; o <<= 1) {
        Run a;
        a.step[0] = __shfl_up_sync(0xFFFFFFFFu, r.step[0], o);
        if (ties) {
            a.step[1] = __shfl_up_sync(0xFFFFFFFFu, r.step[1], o);
            a.out = __shfl_up_sync(0xFFFFFFFFu, r.out, o);
            if (lane >= o) r = run_then(a, r);
        } else if (lane >= o) {
            r.step[0] = wrap_add(a.step[0], r.step[0]);
        }
    }
    return r;
}
__device__ __forceinline__ Run run_from(const Run& r, int src) {
    Run o;
    o.step[0] = __shfl_sync(0xFFFFFFFFu, r.step[0], src);
    o.step[1] = __shfl_sync(0xFFFFFFFFu, r.step[1], src);
    o.out = __shfl_sync(0xFFFFFFFFu, r.out, src);
    return o;
}
__device__ __forceinline__ Run run_identity() { return Run{{0, 0}, 2u}; }

// A step's own run (a step that leaves any binade is marked by the caller).
__device__ __forceinline__ Run run_of(const Step& st) {
    Run r;
    if (st.tie) {
        r.step[0] = st.r + (st.r & 1);
        r.step[1] = st.r + ((1 + st.r) & 1);
        r.out = 0u;
    } else {
        r.step[0] = r.step[1] = st.r;
        r.out = (st.r & 1) ? 1u : 2u;
    }
    return r;
}

// A normal sum's binade: exponent field, sign, and m.
struct Binade {
    int ef, neg;
    long long m;
    bool normal;
};
__device__ __forceinline__ Binade binade_of(double s) {
    const unsigned long long bits = (unsigned long long)__double_as_longlong(s);
    Binade b;
    b.ef = (int)((bits >> 52) & 0x7FF);
    b.neg = (int)(bits >> 63);
    b.m = (long long)(bits & ((1ULL << 52) - 1)) | kM0;
    b.normal = b.ef != 0 && b.ef != 0x7FF;
    return b;
}
__device__ __forceinline__ double sum_of(const Binade& b, long long m) {
    return __longlong_as_double((long long)(((unsigned long long)b.neg << 63) | ((unsigned long long)b.ef << 52) |
                                            (unsigned long long)(m - kM0)));
}
// The value moves no further than a binade's width: its step is a plain integer.
__device__ __forceinline__ bool plain_step(const Step& st) { return !st.fail && st.r < kM1 && st.r > -kM1; }
// The partial m stays strictly inside the binade: then the exact sum it rounds lies in [2^52, 2^53) u
// and was rounded to the binade's ulp (a sum rounding to 2^52 itself may have come from below, where
// the ulp is u / 2).
__device__ __forceinline__ bool inside(long long m) { return m > kM0 && m < kM1; }

struct CtaSum {
    Run warps[kSSThreads / 32];
    int exits[kSSThreads / 32];
    double s;        // the running sum
    int pos;         // values of the block taken
    unsigned alone;  // the block's pieces of 1024 holding an addition taken alone
};

// Whether a value added to a sum that is no normal number may change it: a zero leaves +0 and the
// subnormals as they are, NaN stays, and infinity goes only with NaN or the other infinity.
template <typename T>
__device__ __forceinline__ bool changes_off_binade(double s, T v) {
    if (s != s) return false;
    if (isinf(s)) return v != v || (isinf(v) && (v > (T)0) != (s > 0.0));
    return v != (T)0 || __double_as_longlong(s) == (long long)(1ULL << 63);
}

// One warp's walk over the block's values from `pos`, 32 at a time, until a window holds no value taken
// alone. Every lane holds the same s and pos.
template <typename T>
__device__ __forceinline__ void warp_windows(const SumIn<T>& in, size_t base, int len, double& s, int& pos,
                                             unsigned& alone) {
    const unsigned FULL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    bool crossed = true;
    while (crossed && pos < len) {
        T v = 0;
        const bool has = pos + lane < len && value_at(in, base + pos + lane, &v);
        const Binade b = binade_of(s);
        bool leaves;
        long long before = b.m, last = b.m;
        if (b.normal) {
            Step st{0, 0, 0};
            if (has) st = step_of(v, b.ef, b.neg);
            leaves = !plain_step(st);
            const Run mine = leaves ? run_identity() : run_of(st);
            const Run incl = warp_scan(mine, __any_sync(FULL, st.tie));
            const bool ties = __any_sync(FULL, st.tie);
            const int q = ties ? (int)(b.m & 1) : 0;
            const long long after = wrap_add(b.m, q ? incl.step[1] : incl.step[0]);
            before = __shfl_up_sync(FULL, after, 1);
            if (lane == 0) before = b.m;
            leaves = leaves || (has && v != (T)0 && !inside(after));
            last = __shfl_sync(FULL, after, 31);
        } else {
            leaves = has && changes_off_binade(s, v);
        }
        const unsigned out = __ballot_sync(FULL, leaves);
        if (!out) {
            if (b.normal) s = sum_of(b, last);
            pos += 32;
            crossed = false;
        } else {
            const int e = __ffs(out) - 1;
            const double from = b.normal ? sum_of(b, __shfl_sync(FULL, before, e)) : s;
            s = __shfl_sync(FULL, __dadd_rn(from, (double)v), e);
            alone |= 1u << ((pos + e) / kSSThreads);
            pos += e + 1;
        }
    }
    pos = min(pos, len);
}

// The block's `len` values (a thread's kSSPer consecutive ones in v, its present ones in `has`) added to
// sh.s in order, by the whole CTA. sh.s is set and visible before the call and after it.
template <typename T>
__device__ void cta_advance(const SumIn<T>& in, size_t base, int len, const T (&v)[kSSPer], unsigned has, CtaSum& sh) {
    const unsigned FULL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int first = (int)threadIdx.x * kSSPer;
    int pos = 0;
    if (threadIdx.x == 0) sh.alone = 0;
    while (pos < len) {
        const double s = sh.s;
        const Binade b = binade_of(s);
        const unsigned live = first + kSSPer <= pos ? 0u : first >= pos ? has : has & (0xFFu << (pos - first));
        int exit_at = INT_MAX;
        long long m = b.m, before = 0;   // before: the partial m at this thread's exit
        T vx = 0;
        if (b.normal) {
            long long r[kSSPer];
            unsigned tie = 0, off = 0;
            Run mine = run_identity();
#pragma unroll
            for (int t = 0; t < kSSPer; ++t) {
                Step st{0, 0, 0};
                if (live & (1u << t)) st = step_of(v[t], b.ef, b.neg);
                if (!plain_step(st)) {
                    off |= 1u << t;
                    st = Step{0, 0, 0};
                }
                r[t] = st.r;
                tie |= (unsigned)st.tie << t;
                mine.step[0] = wrap_add(mine.step[0], st.r);
            }
            const bool ties = __syncthreads_or(tie != 0);
            if (ties) {
                mine = run_identity();
#pragma unroll
                for (int t = 0; t < kSSPer; ++t) mine = run_then(mine, run_of(Step{r[t], (int)((tie >> t) & 1u), 0}));
            }
            const Run incl = warp_scan(mine, ties);
            if (lane == 31) sh.warps[warp] = incl;
            __syncthreads();
            const Run wincl = warp_scan(sh.warps[lane], ties);   // every warp scans the warps' totals
            Run start = run_from(wincl, warp > 0 ? warp - 1 : 0);
            if (warp == 0) start = run_identity();
            Run excl;
            excl.step[0] = __shfl_up_sync(FULL, incl.step[0], 1);
            excl.step[1] = __shfl_up_sync(FULL, incl.step[1], 1);
            excl.out = __shfl_up_sync(FULL, incl.out, 1);
            if (lane == 0) excl = run_identity();
            if (ties) {
                start = run_then(start, excl);
                m = wrap_add(m, (b.m & 1) ? start.step[1] : start.step[0]);
            } else {
                m = wrap_add(wrap_add(m, start.step[0]), excl.step[0]);
            }
#pragma unroll
            for (int t = 0; t < kSSPer; ++t) {
                if (exit_at != INT_MAX) continue;
                const long long rt = (tie & (1u << t)) ? r[t] + ((m + r[t]) & 1) : r[t];
                const long long next = wrap_add(m, rt);
                if ((live & (1u << t)) && v[t] != (T)0 && ((off & (1u << t)) || !inside(next))) {
                    exit_at = first + t;
                    before = m;
                    vx = v[t];
                } else {
                    m = next;
                }
            }
        } else {
#pragma unroll
            for (int t = 0; t < kSSPer; ++t)
                if (exit_at == INT_MAX && (live & (1u << t)) && changes_off_binade(s, v[t])) {
                    exit_at = first + t;
                    vx = v[t];
                }
        }
        const int wmin = __reduce_min_sync(FULL, exit_at);
        if (lane == 0) sh.exits[warp] = wmin;
        __syncthreads();
        const int at = __reduce_min_sync(FULL, sh.exits[lane]);
        if (at == INT_MAX) {
            if (threadIdx.x == kSSThreads - 1 && b.normal) sh.s = sum_of(b, m);
            pos = len;
        } else {
            if (exit_at == at) {
                sh.s = __dadd_rn(b.normal ? sum_of(b, before) : s, (double)vx);
                sh.alone |= 1u << (at / kSSThreads);
            }
            __syncthreads();
            if (warp == 0) {
                double t = sh.s;
                int p = at + 1;
                unsigned alone = 0;
                warp_windows(in, base, len, t, p, alone);
                if (lane == 0) {
                    sh.s = t;
                    sh.pos = p;
                    sh.alone |= alone;
                }
            }
            __syncthreads();
            pos = sh.pos;
        }
        __syncthreads();   // sh.s and sh.pos are read before the next scan writes them
    }
}

// A thread's kSSPer consecutive values of the block at `base`: the bits of the present ones.
template <typename T>
__device__ __forceinline__ unsigned load_values(const SumIn<T>& in, size_t base, T (&v)[kSSPer]) {
    unsigned has = 0;
    const size_t i0 = base + (size_t)threadIdx.x * kSSPer;
#pragma unroll
    for (int t = 0; t < kSSPer; ++t) {
        v[t] = 0;
        if (value_at(in, i0 + t, &v[t])) has |= 1u << t;
    }
    return has;
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

// Sums of few blocks, a CTA each, from the first value to the last; the next block's values are loaded
// while this one's are added.
template <typename T>
__global__ void __launch_bounds__(kSSThreads) k_ss_direct(SumJobs<T> jobs) {
    __shared__ CtaSum sh;
    const SumIn<T>& in = jobs.in[blockIdx.x];
    if (threadIdx.x == 0) sh.s = in.init ? *in.init : 0.0;
    __syncthreads();
    long long whole = 0, reduced = 0, alone = 0;
    T v[kSSPer];
    unsigned has = load_values(in, 0, v);
    for (size_t base = 0; base < in.n; base += kSSBlock) {
        T nv[kSSPer];
        const unsigned nhas = load_values(in, base + kSSBlock, nv);
        cta_advance(in, base, (int)(in.n - base < (size_t)kSSBlock ? in.n - base : (size_t)kSSBlock), v, has, sh);
        if (threadIdx.x == 0) {
            const int a = __popc(sh.alone);
            whole += a == 0;
            reduced += a ? kSSPer - a : 0;
            alone += a;
        }
        __syncthreads();   // sh.alone is read before the next block clears it
#pragma unroll
        for (int t = 0; t < kSSPer; ++t) v[t] = nv[t];
        has = nhas;
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
            if (v[t] != (T)0) lw.w.zero = 0;
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
                const bool zero = k < blocks && w.zero && __double_as_longlong(s) != (long long)(1ULL << 63);
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
        T v[kSSPer];
        const unsigned has = load_values(in, base, v);
        cta_advance(in, base, (int)(in.n - base < (size_t)kSSBlock ? in.n - base : (size_t)kSSBlock), v, has, sh);
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
