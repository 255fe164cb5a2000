// Sequential double sums inside a binade as an integer scan (cg_seqsum.cu says why that is exact): the
// device code a CTA walks a block of values with, shared by the sums of cg_seqsum.cu and the sea-level
// cut's histogram walk (cg_cut.cu).
#pragma once

#include <climits>
#include <cstdint>

#include "cg_common.cuh"

namespace cg {
namespace seqwalk {

constexpr int kSSThreads = 1024;
constexpr int kSSPer = 8;                        // values per thread in the parallel reduction
constexpr int kSSBlock = kSSThreads * kSSPer;    // values per block
constexpr long long kM0 = 1LL << 52, kM1 = 1LL << 53;

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

// The value at i; false where it adds nothing: an absent value (a masked cell, which the reference skips)
// or a zero (no sum here is ever -0). The tests are on the values' bits: a double compare is FP64 work.
__device__ __forceinline__ bool value_at(const SumIn<float>& in, size_t i, float* v) {
    if (i >= in.n) return false;
    if (in.mask && !in.mask[i]) return false;
    const float x = in.x[i];
    *v = in.mode == 1 ? __fsub_rn(1.0f, __fmul_rn(0.5f, x)) : x;
    return (__float_as_uint(*v) << 1) != 0;
}

__device__ __forceinline__ bool value_at(const SumIn<double>& in, size_t i, double* v) {
    if (i >= in.n) return false;
    *v = in.x[i];
    return ((unsigned long long)__double_as_longlong(*v) << 1) != 0;
}

// One value's step in the binade with exponent field ef (u = 2^(ef - 1075)), for a sum of sign `neg`:
// the step r when it is not a tie, else the tie's floor f (r = f + ((parity + f) & 1)).
struct Step {
    long long r;
    int tie, fail;
};

// y = M 2^k, M >= 0, negated if asked: fails past 2^kmax M, else rounds to an integer.
__device__ __forceinline__ Step step_from(unsigned long long M, int k, int kmax, bool negative) {
    Step s{0, 0, 0};
    if (k >= 0) {
        s.fail = k > kmax;
        s.r = s.fail ? 0 : (long long)(M << k);
        if (negative) s.r = -s.r;
        return s;
    }
    const int sh = -k < 63 ? -k : 63;   // from 55 on M 2^-sh is below a half
    const unsigned long long rest = M << (64 - sh), half = 1ULL << 63;
    const long long r = (long long)(M >> sh) + (rest > half ? 1 : 0);
    s.tie = rest == half;
    s.r = negative ? -r - s.tie : r;    // a tie's floor
    return s;
}

__device__ __forceinline__ Step step_of(float v, int ef, int neg) {
    const uint32_t b = __float_as_uint(v);
    const int fe = (int)((b >> 23) & 0xFF);
    if (fe == 0xFF) return Step{0, 0, 1};
    const uint32_t M = (b & 0x7FFFFFu) | (fe != 0 ? 1u << 23 : 0u);
    // y = M 2^k with k = (max(fe, 1) - 150) - (ef - 1075); y's sign: x's, flipped for a negative sum
    return step_from(M, (fe == 0 ? 1 : fe) - 150 - ef + 1075, 29, (int)(b >> 31) != neg);
}

// The same for a double value: M < 2^53 and k = max(fe, 1) - ef. NaN, infinity and values of 2^58 u or
// more fail.
__device__ __forceinline__ Step step_of(double v, int ef, int neg) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const int fe = (int)((b >> 52) & 0x7FF);
    if (fe == 0x7FF) return Step{0, 0, 1};
    const unsigned long long M = (b & ((1ULL << 52) - 1)) | (fe != 0 ? 1ULL << 52 : 0ULL);
    return step_from(M, (fe == 0 ? 1 : fe) - ef, 5, (int)(b >> 63) != neg);
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
    double below;    // STOP: the sum before the value that reached the stop
    int hit;         // STOP: that value's index (set to -1 by the caller; -1: none has)
    int pos;         // values of the block taken
    unsigned alone;  // the block's pieces of 1024 holding an addition taken alone
};

// Whether a nonzero value added to a sum that is no normal number may change it: NaN stays, and infinity
// goes only with NaN or the other infinity.
template <typename T>
__device__ __forceinline__ bool changes_off_binade(double s, T v) {
    if (s != s) return false;
    if (isinf(s)) return v != v || (isinf(v) && (v > (T)0) != (s > 0.0));
    return true;
}

// A non-negative sum against a stop >= 0, on the integer pipes: such doubles order as their bits.
__device__ __forceinline__ bool reached(double s, double stop) {
    return __double_as_longlong(s) >= __double_as_longlong(stop);
}

// One warp's walk over the block's values from `pos`, 32 at a time, until a window holds no value taken
// alone. Every lane holds the same s and pos. STOP (sums of values >= 0): the walk ends at the first
// value that brings the sum to `stop`, its index in `hit` and the sum before it in `below`.
template <bool STOP, typename T>
__device__ __forceinline__ void warp_windows(const SumIn<T>& in, size_t base, int len, double& s, int& pos,
                                             unsigned& alone, double stop, int& hit, double& below) {
    const unsigned FULL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    bool crossed = true;
    while (crossed && pos < len) {
        T v = 0;
        const bool has = pos + lane < len && value_at(in, base + pos + lane, &v);
        const Binade b = binade_of(s);
        bool leaves = false;
        long long before = b.m, last = b.m;
        if (b.normal) {
            Step st{0, 0, 0};
            if (has) st = step_of(v, b.ef, b.neg);
            leaves = !plain_step(st);
            const bool ties = __any_sync(FULL, st.tie);
            const Run incl = warp_scan(leaves ? run_identity() : run_of(st), ties);
            const long long after = wrap_add(b.m, ties && (b.m & 1) ? incl.step[1] : incl.step[0]);
            before = __shfl_up_sync(FULL, after, 1);
            if (lane == 0) before = b.m;
            leaves = leaves || (has && (!inside(after) || (STOP && reached(sum_of(b, after), stop))));
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
            if (STOP && reached(s, stop)) {
                hit = pos + e;
                below = from;
                return;
            }
            pos += e + 1;
        }
    }
    pos = min(pos, len);
}

// The CTA's scan of the values [pos, end) of the block, PER consecutive ones a thread from `first`
// (the block's start or pos), under the binade sh.s is in: the index of the first value to be taken
// alone (INT_MAX: none), the sum before it or after the last value, and that value where it is this
// thread's. Every thread calls it; *mine says whether the value is this thread's.
template <int PER, bool STOP, typename T>
__device__ __forceinline__ int cta_scan(const SumIn<T>& in, size_t base, int first, int pos, int end, double s, double stop,
                                        CtaSum& sh, bool* mine, double* from, T* value) {
    const unsigned FULL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int at0 = first + (int)threadIdx.x * PER;
    const Binade b = binade_of(s);
    int exit_at = INT_MAX;
    long long before = b.m, m_end = b.m;
    T vx = 0;
    if (b.normal) {
        long long r[PER], sum = 0, reach = PER;   // reach: how far the thread's partial sums can go, ties' units included
        unsigned has = 0, tie = 0, off = 0;
#pragma unroll
        for (int t = 0; t < PER; ++t) {
            T v;
            r[t] = 0;
            if (at0 + t >= pos && at0 + t < end && value_at(in, base + at0 + t, &v)) {
                const Step st = step_of(v, b.ef, b.neg);
                has |= 1u << t;
                if (plain_step(st)) {
                    r[t] = st.r;
                    tie |= (unsigned)st.tie << t;
                } else {
                    off |= 1u << t;
                }
            }
            sum = wrap_add(sum, r[t]);
            reach = wrap_add(reach, r[t] < 0 ? -r[t] : r[t]);
        }
        const bool ties = __syncthreads_or(tie != 0);
        Run run = run_identity();
        run.step[0] = sum;
        if (ties) {
            run = run_identity();
#pragma unroll
            for (int t = 0; t < PER; ++t) run = run_then(run, run_of(Step{r[t], (int)((tie >> t) & 1u), 0}));
        }
        const Run incl = warp_scan(run, ties);
        if (lane == 31) sh.warps[warp] = incl;
        __syncthreads();
        const Run wincl = warp_scan(sh.warps[lane], ties);   // every warp scans the warps' totals
        const int src = warp > 0 ? warp - 1 : 0;
        Run start = run_identity(), excl = run_identity();
        start.step[0] = __shfl_sync(FULL, wincl.step[0], src);
        excl.step[0] = __shfl_up_sync(FULL, incl.step[0], 1);
        if (ties) {
            start = run_from(wincl, src);
            excl.step[1] = __shfl_up_sync(FULL, incl.step[1], 1);
            excl.out = __shfl_up_sync(FULL, incl.out, 1);
        }
        if (warp == 0) start = run_identity();
        if (lane == 0) excl = run_identity();
        long long m = b.m;
        if (ties) {
            start = run_then(start, excl);
            m = wrap_add(m, (b.m & 1) ? start.step[1] : start.step[0]);
            m_end = wrap_add(m, (m & 1) ? run.step[1] : run.step[0]);
        } else {
            m = wrap_add(wrap_add(m, start.step[0]), excl.step[0]);
            m_end = wrap_add(m, sum);
        }
        // A thread whose partial sums cannot leave the binade (nearly every one) need not walk them.
        if (has && (off || !inside(wrap_add(m, -reach)) || !inside(wrap_add(m, reach)) ||
                    (STOP && reached(sum_of(b, wrap_add(m, reach)), stop)))) {
#pragma unroll
            for (int t = 0; t < PER; ++t) {
                if (exit_at != INT_MAX || !(has & (1u << t))) continue;
                const long long next = wrap_add(m, (tie & (1u << t)) ? r[t] + ((m + r[t]) & 1) : r[t]);
                if ((off & (1u << t)) || !inside(next) || (STOP && reached(sum_of(b, next), stop))) {
                    exit_at = at0 + t;
                    before = m;
                } else {
                    m = next;
                }
            }
            if (exit_at != INT_MAX) value_at(in, base + exit_at, &vx);
        }
    } else {
        for (int t = 0; t < PER && exit_at == INT_MAX; ++t)
            if (at0 + t >= pos && at0 + t < end && value_at(in, base + at0 + t, &vx) && changes_off_binade(s, vx))
                exit_at = at0 + t;
    }
    const int wmin = __reduce_min_sync(FULL, exit_at);
    if (lane == 0) sh.exits[warp] = wmin;
    __syncthreads();
    const int at = __reduce_min_sync(FULL, sh.exits[lane]);
    *mine = at == INT_MAX ? threadIdx.x == kSSThreads - 1 : exit_at == at;
    *from = b.normal ? sum_of(b, at == INT_MAX ? m_end : before) : s;
    *value = vx;
    return at;
}

// The block's `len` values added to sh.s in order, by the whole CTA: a scan of 8 values a thread; from
// a value taken alone on, one warp's windows and then scans of a value a thread, until 1024 values hold
// none. sh.s is set and visible before the call and after it. STOP: as in warp_windows, through sh.hit
// and sh.below.
template <bool STOP = false, typename T>
__device__ void cta_advance(const SumIn<T>& in, size_t base, int len, CtaSum& sh, double stop = 0.0) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int pos = 0;
    bool wide = true;
    if (threadIdx.x == 0) sh.alone = 0;
    while (pos < len) {
        const double s = sh.s;
        const int end = wide ? len : min(len, pos + kSSThreads);
        bool mine;
        double from;
        T value;
        const int at = wide ? cta_scan<kSSPer, STOP>(in, base, 0, pos, end, s, stop, sh, &mine, &from, &value)
                            : cta_scan<1, STOP>(in, base, pos, pos, end, s, stop, sh, &mine, &from, &value);
        if (at == INT_MAX) {
            if (mine) sh.s = from;
            pos = end;
            wide = true;
        } else {
            if (mine) {
                const double to = __dadd_rn(from, (double)value);
                sh.s = to;
                sh.alone |= 1u << (at / kSSThreads);
                if (STOP && reached(to, stop)) {
                    sh.hit = at;
                    sh.below = from;
                }
            }
            __syncthreads();
            if (STOP && sh.hit >= 0) return;
            if (warp == 0) {
                double t = sh.s;
                int p = at + 1;
                unsigned alone = 0;
                int hit = -1;
                double below = 0.0;
                warp_windows<STOP>(in, base, len, t, p, alone, stop, hit, below);
                if (lane == 0) {
                    if (STOP && hit >= 0) {
                        sh.hit = hit;
                        sh.below = below;
                    }
                    sh.s = t;
                    sh.pos = p;
                    sh.alone |= alone;
                }
            }
            __syncthreads();
            if (STOP && sh.hit >= 0) return;
            pos = sh.pos;
            wide = false;
        }
        __syncthreads();   // sh.s and sh.pos are read before the next scan writes them
    }
}

// A thread's kSSPer consecutive values of the block at `base`: the bits of those that add something.
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

}  // namespace seqwalk
}  // namespace cg
