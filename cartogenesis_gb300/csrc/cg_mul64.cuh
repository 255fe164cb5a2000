// IEEE double multiplication on the integer pipes.
//
// GB300 holds a partition's FP64 unit 64 cycles for every warp instruction (77 with all four partitions
// busy), and issues an integer one nearly every cycle: a double product put together from four 32 x 32
// products takes about half the FP64 unit's time and leaves the unit free for additions. The result is
// the product rounded to nearest even, bit for bit, for operands that are zero or normal and products
// that are zero or normal; `Factor::plain` tells which operands those are for twiddle factors.
#pragma once

#include <stdint.h>

#include "cg_fpemu.h"

namespace cg {

// An operand taken apart: its significand shifted up by `kUp` bits (hidden bit included), its exponent
// field and its words.
template <int kUp>
struct Factor {
    uint32_t m1, m0, hi;
    int e;
    CG_HD explicit Factor(double x) {
        const uint64_t b = (uint64_t)fp_bits(x);
        hi = (uint32_t)(b >> 32);
        const uint32_t lo = (uint32_t)b;
        const uint32_t hidden = 1u << (20 + kUp);
        m1 = (((hi << kUp) | (lo >> (32 - kUp))) & (hidden - 1u)) | hidden;
        m0 = lo << kUp;
        e = (int)((hi >> 20) & 0x7FFu);
    }
    CG_HD bool zero() const { return e == 0; }
};
using Value = Factor<11>;
using Weight = Factor<10>;

// Whether value * weight is Factor arithmetic's for every weight of magnitude 0 or 2^-54..1: the value
// is zero, or normal and at least 2^-967, so that no product is subnormal.
CG_HD bool plain_value(double x) {
    const uint64_t b = (uint64_t)fp_bits(x) << 1;
    return b == 0 || ((b >> 53) - 56u) < 2047u - 56u;
}

// The significands are 53 bits up by 11 and 53 up by 10, so the product's upper 64 bits hold 62 or 63:
// 53 to keep and the rest, with a sticky bit for the lower 64, to round.
CG_HD double product(const Value& a, const Weight& b) {
    const uint64_t t = (uint64_t)a.m0 * b.m0;
    const uint64_t u = (uint64_t)a.m1 * b.m0 + (t >> 32);
    const uint64_t v = (uint64_t)a.m0 * b.m1 + (uint32_t)u;
    uint64_t h = (uint64_t)a.m1 * b.m1 + (u >> 32) + (v >> 32);
    h |= ((uint32_t)v | (uint32_t)t) != 0u;
    const uint32_t n = (uint32_t)(h >> 62);   // 1: the significands' product is at least 2
    const uint32_t s = 9u + n;
    const uint64_t q = (h + (uint64_t)(255u + (n << 8) + (((uint32_t)h >> s) & 1u))) >> s;   // half to even
    const uint32_t sign = (a.hi ^ b.hi) & 0x80000000u;
    const bool zero = a.zero() || b.zero();
    // The significand's hidden bit, and a carry out of its rounding, go into the exponent field.
    const uint32_t hi = sign | (zero ? 0u : (uint32_t)(q >> 32) + ((uint32_t)(a.e + b.e - 1024 + (int)n) << 20));
    const uint32_t lo = zero ? 0u : (uint32_t)q;
    return fp_of((int64_t)(((uint64_t)hi << 32) | lo));
}

}  // namespace cg
