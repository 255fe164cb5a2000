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
constexpr int kMostAlone = 512;                  // values of a block cta_segments takes alone, at most
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

// A thread's kSSPer consecutive values of the block at `base`: the bits of those that add something. Whole
// runs of 16-byte aligned values by 16-byte loads: a load a value left 32 bytes between the lanes'.
__device__ __forceinline__ void load_run(const float* x, float (&v)[kSSPer]) {
    const float4 a = reinterpret_cast<const float4*>(x)[0], b = reinterpret_cast<const float4*>(x)[1];
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
}
__device__ __forceinline__ void load_run(const double* x, double (&v)[kSSPer]) {
#pragma unroll
    for (int t = 0; t < kSSPer / 2; ++t) {
        const double2 a = reinterpret_cast<const double2*>(x)[t];
        v[2 * t] = a.x, v[2 * t + 1] = a.y;
    }
}
__device__ __forceinline__ bool adds(const SumIn<float>& in, float& v) {
    if (in.mode == 1) v = __fsub_rn(1.0f, __fmul_rn(0.5f, v));
    return (__float_as_uint(v) << 1) != 0;
}
__device__ __forceinline__ bool adds(const SumIn<double>&, double& v) {
    return ((unsigned long long)__double_as_longlong(v) << 1) != 0;
}
template <typename T>
__device__ __forceinline__ unsigned load_values(const SumIn<T>& in, size_t base, T (&v)[kSSPer]) {
    unsigned has = 0;
    const size_t i0 = base + (size_t)threadIdx.x * kSSPer;
    if (i0 + kSSPer <= in.n && ((uintptr_t)in.x & 15) == 0 && ((uintptr_t)in.mask & 7) == 0) {
        load_run(in.x + i0, v);
        uint2 m = make_uint2(0x01010101u, 0x01010101u);
        if (in.mask) m = *reinterpret_cast<const uint2*>(in.mask + i0);
#pragma unroll
        for (int t = 0; t < kSSPer; ++t)
            if ((((t < 4 ? m.x : m.y) >> (8 * (t & 3))) & 0xFFu) && adds(in, v[t])) has |= 1u << t;
        return has;
    }
#pragma unroll
    for (int t = 0; t < kSSPer; ++t) {
        v[t] = 0;
        if (value_at(in, i0 + t, &v[t])) has |= 1u << t;
    }
    return has;
}
// The bits of a thread's values with indices in [pos, end) of the block.
__device__ __forceinline__ unsigned within(int pos, int end) {
    const int lo = pos - (int)threadIdx.x * kSSPer, hi = end - (int)threadIdx.x * kSSPer;
    const unsigned below_hi = hi >= kSSPer ? 0xFFu : (hi <= 0 ? 0u : (1u << hi) - 1u);
    const unsigned below_lo = lo >= kSSPer ? 0xFFu : (lo <= 0 ? 0u : (1u << lo) - 1u);
    return below_hi & ~below_lo;
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
    // cta_segments: the values taken alone in order, the steps of all others before each, and the binade
    // (exponent | sign << 11, -1: no value) of the others between it and the one before.
    long long steps[kMostAlone + 1];
    double values[kMostAlone];
    int at[kMostAlone], spec[kMostAlone + 1];
    int odd;         // cta_classify: steps more from an odd start
    long long totals[kSSThreads / 32];
    int counts[kSSThreads / 32];
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

// Values that cross one after another: the next `run` of the block added in hardware, one after another, by a
// warp. A window that ends at a value taken alone costs some 0.5 us, an addition 40 ns, so this follows a
// window that ended within kFewSteps values, with runs that double while it stays so. With windows alone 2^21
// values of alternating sign took 1040 ms, 93 so (pieces of 1024 added by one thread from shared memory:
// 151 for floats, 90 for doubles).
constexpr int kFewSteps = 12, kLeastAlone = 64, kMostRun = 1024;
template <typename T>
__device__ __forceinline__ void warp_alone(const SumIn<T>& in, size_t base, int len, int run, double& s, int& pos,
                                           unsigned& alone) {
    const unsigned FULL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31, end = min(len, pos + run);
    for (; pos < end; pos += 32) {
        T v = 0;
        const bool has = pos + lane < end && value_at(in, base + pos + lane, &v);
        const unsigned here = __ballot_sync(FULL, has);
        const double d = has ? (double)v : 0.0;   // a zero adds nothing: no sum here is ever -0
#pragma unroll
        for (int j = 0; j < 32; ++j) s = __dadd_rn(s, __shfl_sync(FULL, d, j));
        if (here) alone |= 1u << ((pos + __ffs(here) - 1) / kSSThreads) | 1u << ((pos + 31 - __clz(here)) / kSSThreads);
    }
    pos = min(pos, end);
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
    int run = kLeastAlone;
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
            if (!STOP && e < kFewSteps) {
                warp_alone(in, base, len, run, s, pos, alone);
                run = min(2 * run, kMostRun);
            } else {
                run = kLeastAlone;
            }
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
        // Floats as a run (`first` is the block's start); doubles one by one, a run of them takes registers
        // the scan has not got (35 us a book's seven blocks against 46).
        constexpr bool kRun = PER == kSSPer && sizeof(T) == 4;
        T x[kRun ? kSSPer : 1];
        if constexpr (kRun) has = load_values(in, base, x) & within(pos, end);
#pragma unroll
        for (int t = 0; t < PER; ++t) {
            r[t] = 0;
            T& v = x[kRun ? t : 0];
            if (kRun ? (has >> t) & 1u : at0 + t >= pos && at0 + t < end && value_at(in, base + at0 + t, &v)) {
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

// A magnitude and its exponent: |v| = M 2^e, M < 2^53 (2^24 for floats).
struct Magnitude {
    unsigned long long M;
    int e;
    bool neg, finite;
};
__device__ __forceinline__ Magnitude magnitude_of(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const int fe = (int)((b >> 52) & 0x7FF);
    return Magnitude{(b & (kM0 - 1)) | (fe != 0 ? (unsigned long long)kM0 : 0ull), (fe == 0 ? 1 : fe) - 1075, (b >> 63) != 0,
                     fe != 0x7FF};
}
__device__ __forceinline__ Magnitude magnitude_of(float v) {
    const uint32_t b = __float_as_uint(v);
    const int fe = (int)((b >> 23) & 0xFF);
    return Magnitude{(b & 0x7FFFFFu) | (fe != 0 ? 1u << 23 : 0u), (fe == 0 ? 1 : fe) - 150, (b >> 31) != 0, fe != 0xFF};
}
// The exponent field's width, and a value's (nonzero values; 0: subnormal).
template <typename T>
constexpr int kTopField = sizeof(T) == 8 ? 0x7FF : 0xFF;
__device__ __forceinline__ int field_of(double v) { return (__double2hiint(v) >> 20) & 0x7FF; }
__device__ __forceinline__ int field_of(float v) { return (int)((__float_as_uint(v) >> 23) & 0xFF); }
// The binary exponent of a nonzero magnitude: 2^x <= |v| < 2^(x + 1).
__device__ __forceinline__ int exponent_of(const Magnitude& a) { return a.e + 63 - __clzll((long long)a.M); }
// v in units of 2^unit, toward zero: off by less than a unit. |v| < 2^(unit + 61).
__device__ __forceinline__ long long units_of(const Magnitude& a, int unit) {
    const int up = a.e - unit;
    const unsigned long long q = up >= 0 ? a.M << up : (up > -64 ? a.M >> -up : 0ull);
    return a.neg ? -(long long)q : (long long)q;
}

// An int64 scan over the CTA: *before receives the values before this thread's, the result is
// the total. `totals` is free again after the next barrier.
__device__ __forceinline__ long long cta_before(long long v, long long* before, long long* totals) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    long long x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x = wrap_add(x, y);
    }
    if (lane == 31) totals[warp] = x;
    __syncthreads();
    long long w = totals[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long y = __shfl_up_sync(0xFFFFFFFFu, w, o);
        if (lane >= o) w = wrap_add(w, y);
    }
    const long long start = __shfl_sync(0xFFFFFFFFu, w, warp > 0 ? warp - 1 : 0);
    *before = wrap_add(warp > 0 ? start : 0, wrap_add(x, -v));
    return __shfl_sync(0xFFFFFFFFu, w, 31);
}

// What is known of the parity of a sum's m: even, odd, that of the sum the block starts from or the other
// one, or nothing; and what a run of values makes of it, a parity or (kParityKeep, + 1: the other one) a
// change of it. A tie leaves m even, whatever it was.
using Parity = int;
constexpr Parity kParityEven = 0, kParityStart = 2, kParityUnknown = 4, kParityKeep = 8;
__device__ __forceinline__ Parity parity_then(Parity a, Parity b) {
    if (b < kParityKeep) return b;
    return a == kParityUnknown ? a : a ^ (b & 1);   // of a change: the changes add up
}
// A tie's step from a sum of parity `state` (of an even start), and how much more it is from an odd start.
__device__ __forceinline__ long long tie_value(const Step& st, Parity state) { return st.r + (((state & 1) + st.r) & 1); }
__device__ __forceinline__ bool tie_step(const Step& st, Parity state, long long* odd) {
    *odd = (state & 2) ? tie_value(st, state ^ 1) - tie_value(st, state) : 0;
    return state != kParityUnknown;
}

// The block's values [pos, len) after a sum of about `start`, crossings and all, told apart: the values to be
// taken alone are listed in sh (steps, values, at, spec), and the steps of all others summed. The partial
// sums are first taken in fixed point, in units of 2^-60 of what they can reach, by one integer scan: they
// are off from the rounded sums by less than 2^20 units (a unit a value, and the rounded sums' own
// roundings, 2^6 units each) and what `start` is off (`start_off`), which tells each partial sum's binade
// but next to a power of two. A value whose sums before and after are surely in one binade is a step of that
// binade, whatever the parity unless it is a tie; a tie's step follows from the parity, which is known from
// the tie before it on (a scan of the parities, where there are ties), is `entry`'s at the block's start, and
// is not known after a crossing. Every other value is listed. The steps are taken for a block that starts
// even; sh.odd is what one that starts odd takes more, before the first listed value. The steps between two
// listed values are a difference of a second scan. Returns how many values are listed, or -1 where that does not
// apply: a sum or value that is not finite, or too many values; *all_steps receives the steps of the rest.
// Every thread calls it, and what it wrote to sh is visible after it.
template <bool STOP, typename T>
__device__ int cta_classify(const SumIn<T>& in, size_t base, int pos, int len, double start, double start_off, Parity entry,
                            CtaSum& sh, double stop, long long* all_steps) {
    const unsigned FULL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int at0 = (int)threadIdx.x * kSSPer;
    const Magnitude ms = magnitude_of(start), mo = magnitude_of(start_off);
    T v[kSSPer];
    const unsigned has = load_values(in, base, v) & within(pos, len);
    // The largest exponent field, and so whether every value is finite.
    int top = -1;
#pragma unroll
    for (int t = 0; t < kSSPer; ++t)
        if ((has >> t) & 1u) top = max(top, field_of(v[t]));
    top = __reduce_max_sync(FULL, top);
    if (lane == 0) sh.counts[warp] = top;
    for (int k = threadIdx.x; k <= kMostAlone; k += kSSThreads) sh.spec[k] = -1;
    if (threadIdx.x == 0) sh.odd = 0;
    __syncthreads();
    top = __reduce_max_sync(FULL, sh.counts[lane]);
    *all_steps = 0;
    if (!ms.finite || !mo.finite || top == kTopField<T>) return -1;
    if (top < 0) return 0;   // nothing to add
    // |every partial sum| < 2^(reach + 1): the sum before and 2^13 values.
    const int most = max(top, 1) - kTopField<T> / 2;   // the largest value's binary exponent
    const int reach = max(max(ms.M ? exponent_of(ms) : INT_MIN, mo.M ? exponent_of(mo) : INT_MIN) + 1, most + 13) + 1;
    const int unit = reach - 59;
    const long long off = (1ll << 20) + units_of(mo, unit) + 1;   // < 2^59
    long long stop_units = 0;
    if (STOP) {
        const Magnitude a = magnitude_of(stop);
        stop_units = a.M && exponent_of(a) > reach ? LLONG_MAX / 2 : units_of(a, unit);
    }
    long long sum = 0, span = 0, before;   // span: how far this thread's values can go
#pragma unroll
    for (int t = 0; t < kSSPer; ++t) {
        const long long q = (has >> t) & 1u ? units_of(magnitude_of(v[t]), unit) : 0;
        sum += q;
        span += q < 0 ? -q : q;
    }
    cta_before(sum, &before, sh.totals);
    const long long p0 = units_of(ms, unit) + before;
    // The surely known binade of a partial sum: exponent field | sign << 11, or -1.
    auto binade_at = [=](long long p) {
        const long long a = p < 0 ? -p : p;
        const int bit = 63 - __clzll(a);
        if (a <= 4 * off || a - (1ll << bit) <= off || (2ll << bit) - a <= off) return -1;
        const int ef = bit + unit + 1023;
        return ef >= 1 && ef <= 2046 ? ef | (p < 0 ? 1 << 11 : 0) : -1;
    };
    auto near_stop = [=](long long was, long long p) { return STOP && p >= stop_units - 2 * off && was <= stop_units + 2 * off; };
    const int first = binade_at(p0);
    // All of the thread's sums are surely in one binade (nearly every thread's are).
    const bool quiet = first >= 0 && binade_at(p0 - span) == first && binade_at(p0 + span) == first &&
                       !near_stop(p0 - span, p0 + span);
    // The thread's values in order: whether one is to be taken alone, else its step and binade.
    auto each = [&](auto&& take) {
        long long p = p0;
        int code = first;
#pragma unroll
        for (int t = 0; t < kSSPer; ++t) {
            if (!((has >> t) & 1u)) continue;
            int next = code;
            bool alone = false;
            if (!quiet) {
                const long long was = p;
                p += units_of(magnitude_of(v[t]), unit);
                next = binade_at(p);
                alone = code < 0 || next != code || near_stop(was, p);
            }
            Step st{0, 0, 0};
            if (!alone) {
                st = step_of(v[t], code & 0x7FF, code >> 11);
                alone = !plain_step(st);
            }
            take(t, alone, st, code);
            code = next;
        }
    };
    long long steps = 0;
    unsigned single = 0;
    int spec[2] = {-1, -1};   // the binades of this thread's first steps, and of those after its last listed value
    auto note = [&](int t, bool alone, long long step, int code) {
        if (alone) {
            single |= 1u << t;
            spec[1] = -1;
        } else {
            steps = wrap_add(steps, step);
            spec[single ? 1 : 0] = code;
        }
    };
    bool tie = false;
    Parity moves = kParityKeep;
    each([&](int t, bool alone, const Step& st, int code) {
        note(t, alone, st.r, code);
        tie |= !alone && st.tie;
        moves = parity_then(moves, alone ? kParityUnknown : st.tie ? kParityEven : kParityKeep + (int)(st.r & 1));
    });
    Parity enters = entry;
    const bool ties = __syncthreads_or(tie);   // and sh.totals and sh.counts are read
    if (ties) {
        Parity x = moves;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const Parity y = __shfl_up_sync(FULL, x, o);
            if (lane >= o) x = parity_then(y, x);
        }
        if (lane == 31) sh.counts[warp] = x;
        __syncthreads();
        Parity w = sh.counts[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const Parity y = __shfl_up_sync(FULL, w, o);
            if (lane >= o) w = parity_then(y, w);
        }
        w = __shfl_sync(FULL, w, warp > 0 ? warp - 1 : 0);
        x = __shfl_up_sync(FULL, x, 1);
        if (warp > 0) enters = parity_then(enters, w);
        if (lane > 0) enters = parity_then(enters, x);
        steps = 0;
        single = 0;
        spec[0] = spec[1] = -1;
        Parity state = enters;
        each([&](int t, bool alone, const Step& st, int code) {
            long long odd;
            const bool unknown = !alone && st.tie && !tie_step(st, state, &odd);
            if (!alone && st.tie && !unknown && odd != 0) sh.odd = (int)odd;
            note(t, alone || unknown, st.tie && !unknown ? tie_value(st, state) : st.r, code);
            state = parity_then(state, alone ? kParityUnknown : st.tie ? kParityEven : kParityKeep + (int)(st.r & 1));
        });
        __syncthreads();   // sh.counts is read
    }
    long long steps_before;
    *all_steps = cta_before(steps, &steps_before, sh.totals);
    int mine = __popc(single), slot = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FULL, slot, o);
        if (lane >= o) slot += y;
    }
    if (lane == 31) sh.counts[warp] = slot;
    __syncthreads();
    const int c = sh.counts[lane], listed = __reduce_add_sync(FULL, c);
    slot += __reduce_add_sync(FULL, lane < warp ? c : 0) - mine;
    if (listed > kMostAlone) return -1;
    if (spec[0] >= 0) sh.spec[slot] = spec[0];
    if (spec[1] >= 0) sh.spec[slot + mine] = spec[1];
    if (single) {   // the thread's values again, for the steps between its listed ones
        Parity state = enters;
        each([&](int t, bool alone, const Step& st, int) {
            if ((single >> t) & 1u) {
                sh.steps[slot] = steps_before;
                sh.values[slot] = (double)v[t];
                sh.at[slot] = at0 + t;
                ++slot;
            } else {
                steps_before = wrap_add(steps_before, st.tie ? tie_value(st, state) : st.r);
            }
            state = parity_then(state, alone ? kParityUnknown : st.tie ? kParityEven : kParityKeep + (int)(st.r & 1));
        });
    }
    __syncthreads();
    return listed;
}

// The block's values [pos, len) added to sh.s at once: told apart, then chained by one thread, one addition
// in hardware and a few instructions a listed value, about 0.15 us, where a CTA scan for each crossing took
// 3 to 5. The chain checks that a run of steps ends inside a binade, and that it is the one they were taken
// for (but for runs within one thread). Returns false, with sh.s as it was, where that does not apply. sh.s
// is set and visible before the call and after it.
template <bool STOP, typename T>
__device__ bool cta_segments(const SumIn<T>& in, size_t base, int pos, int len, CtaSum& sh, double stop) {
    const double s0 = sh.s;
    long long all_steps;
    const Binade b0 = binade_of(s0);
    const int listed = cta_classify<STOP>(in, base, pos, len, s0, 0.0, b0.normal ? (Parity)(b0.m & 1) : kParityUnknown, sh,
                                          stop, &all_steps);
    if (listed < 0) return false;
    if (threadIdx.x == 0) {
        double s = s0;
        long long done = 0;
        unsigned alone = 0;
        bool sound = true;
        int hit = -1;
        double from = 0.0;
        for (int k = 0; k <= listed; ++k) {
            const long long run = wrap_add(k < listed ? sh.steps[k] : all_steps, -done);
            if (run != 0) {
                const Binade b = binade_of(s);
                const long long m = b.m + run;
                const int spec_k = sh.spec[k];
                sound &= b.normal && inside(m) && (spec_k == -1 || spec_k == (b.ef | (b.neg << 11)));
                s = sum_of(b, m);
                done = wrap_add(done, run);
            }
            if (k == listed) break;
            from = s;
            s = __dadd_rn(s, sh.values[k]);
            alone |= 1u << (sh.at[k] / kSSThreads);
            if (STOP && reached(s, stop)) {
                hit = sh.at[k];
                break;
            }
        }
        sh.pos = sound;
        if (sound) {
            sh.s = s;
            sh.alone |= alone;
            if (STOP && hit >= 0) {
                sh.hit = hit;
                sh.below = from;
            }
        }
    }
    __syncthreads();
    return sh.pos != 0;
}

// The block's `len` values added to sh.s in order, by the whole CTA: a scan of 8 values a thread; from
// a value taken alone on, all the rest at once by their predicted binades, or, where that does not apply,
// one warp's windows and then scans of a value a thread, until 1024 values hold none. sh.s is set and
// visible before the call and after it. STOP: as in warp_windows, through sh.hit and sh.below.
// `crosses`: the caller knows that a scan would not take the block.
template <bool STOP = false, typename T>
__device__ void cta_advance(const SumIn<T>& in, size_t base, int len, CtaSum& sh, bool crosses = false, double stop = 0.0) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int pos = 0;
    bool wide = true, predict = true;
    if (threadIdx.x == 0) sh.alone = 0;
    if (crosses) {
        predict = false;
        if (cta_segments<STOP>(in, base, 0, len, sh, stop)) return;
        __syncthreads();   // sh.pos is read
    }
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
            if (wide && predict) {
                predict = false;   // once a block: what it cannot take, it could not later
                if (cta_segments<STOP>(in, base, at + 1, len, sh, stop)) return;
                __syncthreads();   // sh.pos is read
            }
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

}  // namespace seqwalk
}  // namespace cg
