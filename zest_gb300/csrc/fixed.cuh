// FP64 values to and from 64-bit fixed point by integer operations (the FP64 pipe
// of GB300 retires one operation per 64 of the integer pipe).
#pragma once

#include <cuda_runtime.h>

namespace zgpu {

// 2^E T for a signed 64-bit T, rounded to nearest even, without FP64 operations
// and without branches (so that independent elements interleave), in 32-bit
// halves: |T| below 2^32 is moved
// up by 32 bits first, so that one 32-bit leading-zero count and two funnel
// shifts normalise it; the rounding carry runs into the exponent field through
// the bit pattern; zero, results below the normal range and overflow are
// selected at the end.
__device__ __forceinline__ double i64_ldexp(long long T, int E) {
    const unsigned long long sm = (unsigned long long)(T >> 63);  // all ones for T < 0
    const unsigned long long a = ((unsigned long long)T ^ sm) - sm;
    const bool small = (a >> 32) == 0;
    const unsigned ah = small ? (unsigned)a : (unsigned)(a >> 32);
    const unsigned al = small ? 0u : (unsigned)a;
    const int lz = __clz(ah);                           // 32 only for T = 0
    const unsigned nh = __funnelshift_l(al, ah, lz);    // leading one at bit 31
    const unsigned nl = al << (lz & 31);
    const unsigned mh = nh >> 11;                       // mantissa bits 52..32 (the leading one at bit 20)
    const unsigned ml = __funnelshift_r(nl, nh, 11);    // mantissa bits 31..0
    const unsigned inc = ((nl & 0x7FFu) + (ml & 1u) + 0x3FFu) >> 11;  // round half to even
    const int e = E + 1023 + 63 - (small ? 32 : 0) - lz;  // exponent field of the leading one
    const unsigned lo = ml + inc;
    const unsigned mc = mh + (lo < ml ? 1u : 0u);
    const int eff = e + int(mc >> 21);                  // after a rounding carry
    const unsigned hi = (eff >= 2047 ? 0x7FF00000u : ((unsigned)(e - 1) << 20) + mc) |
                        ((unsigned)(sm >> 32) & 0x80000000u);
    const double v = __hiloint2double((int)hi, eff >= 2047 ? 0 : (int)lo);
    return (a == 0 || eff <= 0) ? 0.0 : v;
}

// The same for a result that is zero or in the normal range whatever T is
// (-1022 <= E <= 958): no selects for the ends of the range, the rounding as one
// carry chain from the dropped bits into the exponent, and the shift amounts
// folded into the exponent by a multiply-add: 22 integer-pipe operations
// where the form above takes 38.  base = (E + 1085) 2^20.
__device__ __forceinline__ double i64_ldexp_normal(long long T, int base) {
    const int sm = int(T >> 63);
    const unsigned long long sm2 = (unsigned long long)(long long)sm;
    const unsigned long long a = ((unsigned long long)T ^ sm2) - sm2;
    const bool small = (a >> 32) == 0;
    const unsigned ah = small ? (unsigned)a : (unsigned)(a >> 32);
    const unsigned al = small ? 0u : (unsigned)a;
    const int lz = __clz(ah);
    const unsigned nh = __funnelshift_l(al, ah, lz);  // leading one at bit 31
    const unsigned nl = al << (lz & 31);
    const unsigned mh = nh >> 11, ml = __funnelshift_r(nl, nh, 11);
    const unsigned top = unsigned(base) - (unsigned(lz + (small ? 32 : 0)) << 20);
    // dropped bits at the top, the kept lowest bit below them: a carry out of
    // this sum is a rounding up (half to even)
    const unsigned r = (nl << 21) | (ml & 1u);
    unsigned lo, hi;
    asm("{\n\t.reg .u32 t;\n\tadd.cc.u32 t, %2, 0x7FFFFFFF;\n\taddc.cc.u32 %0, %3, 0;\n\taddc.u32 %1, %4, %5;\n\t}"
        : "=r"(lo), "=r"(hi)
        : "r"(r), "r"(ml), "r"(mh), "r"(top));
    hi |= unsigned(sm) & 0x80000000u;
    return __hiloint2double(int(ah ? hi : 0u), int(lo));
}

// fixed point: round(x 2^{nbits-e}) as int64 (|x| < 2^(e-1)), ties away from
// zero, with Cr = 1074 + e - nbits.  q = |x| 2^{nbits-e+1} truncated (one bit
// more than kept), then ((q ^ s) + 1) >> 1 with s the sign mask is
// floor(q/2 + 1/2) for x >= 0 and its negative for x < 0.  The shift
// Cr - E(x) is at least 5 for every element of a row (the row exponent keeps
// a bit of headroom); PTX shifts of 64 or more give 0, so a zero or an element
// far below the row's largest rounds to 0 without a branch.
// A bias is added with the rounding one.
__device__ __forceinline__ long long to_fixed_c(double x, int Cr, long long bias = 0) {
    const unsigned long long bits = (unsigned long long)__double_as_longlong(x);
    const unsigned E = unsigned(bits >> 52) & 0x7FFu;
    const unsigned long long M = (bits & 0xFFFFFFFFFFFFFull) | (1ull << 52);
    unsigned long long q;
    asm("shr.b64 %0, %1, %2;" : "=l"(q) : "l"(M), "r"(unsigned(Cr) - E));
    const long long sg = (long long)bits >> 63;  // 0 or -1
    return (((long long)q ^ sg) + (1 + 2 * bias)) >> 1;
}

// A fixed-point value as h 2^31 + l with a balanced low limb, |l| <= 2^30.
struct Limbs {
    int h, l;
};
__device__ __forceinline__ Limbs limbs(long long v) {
    const int l = int(unsigned(v) << 1) >> 1;
    return Limbs{int((v - l) >> 31), l};
}
__device__ __forceinline__ long long mad_wide(int a, int b, long long c) {
    long long r;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
}
// Sum of products value x constant, the constants with CBITS fraction bits:
// three 32 x 32 -> 64-bit multiply-adds a term (the product of the low limbs,
// below 2^(60 - CBITS), is dropped), rounded once at the end.  The caller bounds
// the terms: |xl ch| <= 2^(30 + CBITS - 31) each, and sum |xh| 2^30, below 2^63.
template <int CBITS>
struct FixedAcc {
    long long p1 = 0, p2 = 1ll << (CBITS - 32);  // half a unit
    __device__ __forceinline__ void add(Limbs x, int ch, int cl) {
        p1 = mad_wide(x.h, ch, p1);
        p2 = mad_wide(x.h, cl, p2);
        p2 = mad_wide(x.l, ch, p2);
    }
    __device__ __forceinline__ long long value() const {
        return (long long)((unsigned long long)p1 << (62 - CBITS)) + (p2 >> (CBITS - 31));
    }
};

// Scale of a set of values from the high word of the largest magnitude:
// |x| < 2^scale; and whether that is an infinity or a NaN.
__device__ __forceinline__ int fixed_scale(unsigned hi) { return max(int(hi >> 20), 64) - 1022; }
__device__ __forceinline__ bool not_finite(unsigned hi) { return hi >= 0x7FF00000u; }
__device__ __forceinline__ double nan64() { return __longlong_as_double(0x7FF8000000000000ll); }

}  // namespace zgpu
