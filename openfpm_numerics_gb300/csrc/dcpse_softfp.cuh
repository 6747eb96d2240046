// dcpse_softfp.cuh -- FP64 products on the integer pipes.
//
// GB300's FP64 pipe takes 16 SM cycles per warp instruction (2 lanes per cycle
// per SM), whatever the instruction: product, sum, comparison or conversion.
// The same correctly rounded product takes about 33 integer instructions,
// 13.1 SM cycles by itself (152 SMs, 32 warps each, measured against 16-18.7
// for dmul), and runs beside the FP64 pipe: half the products here and half
// there take 9.4 cycles each.  Kernels bound by the FP64 pipe therefore form
// their products here and leave the pipe to the sums.
#pragma once

#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#include "dcpse_common.cuh"
#endif

#if defined(__CUDACC__)
#define DCPSE_HD __host__ __device__ __forceinline__
#else
#define DCPSE_HD inline
#endif

namespace dcpse {

// The words of x, on the device by the intrinsics: integer tests of a bit cast
// (x << 1 == 0) would be compiled to floating comparisons, on the FP64 pipe.
DCPSE_HD uint32_t dhi(double x) {
#ifdef __CUDA_ARCH__
    return (uint32_t)__double2hiint(x);
#else
    uint64_t u;
    std::memcpy(&u, &x, sizeof u);
    return (uint32_t)(u >> 32);
#endif
}
DCPSE_HD uint32_t dlo(double x) {
#ifdef __CUDA_ARCH__
    return (uint32_t)__double2loint(x);
#else
    uint64_t u;
    std::memcpy(&u, &x, sizeof u);
    return (uint32_t)u;
#endif
}
DCPSE_HD bool is_zero(double x) { return ((dhi(x) << 1) | dlo(x)) == 0u; }
DCPSE_HD bool is_plus_zero(double x) { return (dhi(x) | dlo(x)) == 0u; }

DCPSE_HD double from_bits(uint32_t hi, uint32_t lo) {
#ifdef __CUDA_ARCH__
    return __hiloint2double((int)hi, (int)lo);
#else
    const uint64_t u = ((uint64_t)hi << 32) | lo;
    double d;
    std::memcpy(&d, &u, sizeof d);
    return d;
#endif
}

// (hi:lo) >> s, low word, and (hi:lo) << s, high word, 0 <= s < 32
DCPSE_HD uint32_t shr_pair(uint32_t lo, uint32_t hi, uint32_t s) {
#ifdef __CUDA_ARCH__
    return __funnelshift_r(lo, hi, s);
#else
    return (uint32_t)((((uint64_t)hi << 32) | lo) >> s);
#endif
}
DCPSE_HD uint32_t shl_pair(uint32_t lo, uint32_t hi, uint32_t s) {
#ifdef __CUDA_ARCH__
    return __funnelshift_l(lo, hi, s);
#else
    return (uint32_t)(((((uint64_t)hi << 32) | lo) << s) >> 32);
#endif
}

// Whether rn_mul_int takes x: 2^-255 <= |x| < 2^257 (exponent fields 768 to
// 1279: no product of two such numbers comes near the range's ends) ...
DCPSE_HD bool int_range(double x) {
    return ((dhi(x) & 0x7fffffffu) - 0x30000000u) < 0x20000000u;
}
// ... or a zero, which products with such numbers may have on one side
DCPSE_HD bool int_range_or_zero(double x) { return int_range(x) || is_zero(x); }

// RN(a b), bit for bit IEEE round to nearest even, for a and b in int_range or
// zero.  The 106-bit product of the significands, its top 64 bits with a
// sticky bit, normalised by at most one place, rounded at bit 11; the implicit
// one of the result carries into the exponent field.
DCPSE_HD double rn_mul_int(double a, double b) {
    const uint32_t ah = dhi(a), al = dlo(a), bh = dhi(b), bl = dlo(b);
    const uint32_t am = (ah & 0xfffffu) | 0x100000u, bm = (bh & 0xfffffu) | 0x100000u;
    const uint64_t t0 = (uint64_t)al * bl;
    const uint64_t t1 = (uint64_t)al * bm + (t0 >> 32);
    const uint64_t t2 = (uint64_t)am * bl + t1;
    const uint64_t t3 = (uint64_t)am * bm + (t2 >> 32);
    const uint32_t p0 = (uint32_t)t0, p1 = (uint32_t)t2, p2 = (uint32_t)t3, p3 = (uint32_t)(t3 >> 32);
    uint32_t hi = shr_pair(p2, p3, 10), lo = shr_pair(p1, p2, 10);  // bits 42 and up: 63 or 64 of them
    lo |= ((p1 & 0x3ffu) | p0) != 0u;                               // sticky
    const uint32_t n = hi >> 31, s = n ^ 1u;
    hi = shl_pair(lo, hi, s);
    lo <<= s;
    const uint32_t mh = hi >> 11, ml = shr_pair(lo, hi, 11);
    const uint32_t inc = ((lo & 0x7ffu) + (ml & 1u)) > 0x400u;
    const uint32_t es = (ah & 0x7ff00000u) + (bh & 0x7ff00000u);
    const bool zero = es < 0x60000000u;  // two in range add up to at least 1536
    const uint64_t r = (((uint64_t)(es - (1024u << 20) + (n << 20) + mh) << 32) | ml) + inc;
    const uint32_t sign = (ah ^ bh) & 0x80000000u;
    return from_bits(zero ? sign : ((uint32_t)(r >> 32) | sign), zero ? 0u : (uint32_t)r);
}

// RN(a / b) for a (or its zero), b and r in int_range, r within an ulp or two of
// 1 / b: the quotient a r is off by a few ulps at most, and its exact remainder
// A 2^s - B Q (significands as integers; it fits 64 bits, so only its low 64 are
// formed) says which neighbour is nearest (the final-rounding argument of Markstein,
// IBM J. Res. Dev. 34, 1990, in integers; a quotient is never half way).  False,
// for the caller to divide, where the quotient is a power of two from above
// (the spacing changes there) or more than one ulp off.
DCPSE_HD bool rn_div_int(double a, double b, double r, double& q) {
    q = rn_mul_int(a, r);
    if (is_zero(q)) return true;
    const uint32_t ah = dhi(a), bh = dhi(b), qh = dhi(q), ql = dlo(q), bl = dlo(b);
    const uint32_t bm = (bh & 0xfffffu) | 0x100000u, qm = (qh & 0xfffffu) | 0x100000u;
    // exponent of q below that of A / B in [1/2, 2): 0 or 1 (or -1 for a quotient rounded up to 2)
    const int down = (int)((ah >> 20) & 0x7ffu) - (int)((bh >> 20) & 0x7ffu) + 1023 - (int)((qh >> 20) & 0x7ffu);
    const uint64_t num = (uint64_t)(dlo(a) << (20 + down)) << 32;
    int64_t rem = (int64_t)(num - ((uint64_t)bl * ql + ((uint64_t)(bl * qm + bm * ql) << 32)));
    const int64_t B = (int64_t)(((uint64_t)bm << 32) | bl);
    const bool low = qm == 0x100000u && ql == 0u && rem < 0;
    const int up = 2 * rem > B, dn = 2 * rem < -B;
    rem -= up ? B : 0;
    rem += dn ? B : 0;
    const uint64_t bits = ((((uint64_t)qh << 32) | ql) + (uint64_t)(int64_t)(up - dn));
    q = from_bits((uint32_t)(bits >> 32), (uint32_t)bits);
    return 2 * rem <= B && 2 * rem >= -B && !low && !((bits & 0xfffffffffffffull) == 0 && rem < 0);
}

// Whether x is 0 or 2^-16 <= |x| < 2^17: products of up to 8 such factors stay
// within 2^136, and the product of one of those and a number below 2^101 (or a
// zero) in int_range
DCPSE_HD bool unit_range_or_zero(double x) {
    return ((dhi(x) & 0x7fffffffu) - 0x3ef00000u) < 0x02100000u || is_zero(x);
}
// 2^-100 <= |x| < 2^101, or a zero
DCPSE_HD bool coef_range_or_zero(double x) {
    return ((dhi(x) & 0x7fffffffu) - 0x39b00000u) < 0x0c900000u || is_zero(x);
}

// (float)x, round to nearest even, for results that are normal floats
DCPSE_HD bool narrow_range(double x) {  // 2^-126 <= |x| < 2^127
    return ((dhi(x) & 0x7fffffffu) - 0x38100000u) < 0x0fd00000u;
}
DCPSE_HD uint32_t narrow_bits(double x) {
    const uint32_t hi = dhi(x), lo = dlo(x);
    uint32_t r = shr_pair(lo, (hi & 0x7fffffffu) - 0x38000000u, 29);
    r += ((lo & 0x1fffffffu) + (r & 1u)) > 0x10000000u;
    return r | (hi & 0x80000000u);
}
// (double)f of a normal float's bits
DCPSE_HD double widen_bits(uint32_t f) {
    return from_bits(((f & 0x7fffffffu) >> 3) + 0x38000000u + (f & 0x80000000u), f << 29);
}

#if defined(__CUDACC__)
// The FP64 pipe's own instruction on the rare side of a branch, as volatile asm:
// the compiler would otherwise execute it on both sides and select.
__device__ __forceinline__ double pipe_fma(double a, double b, double c) {
    double d;
    asm volatile("fma.rn.f64 %0, %1, %2, %3;" : "=d"(d) : "d"(a), "d"(b), "d"(c));
    return d;
}

// a conversion costs the FP64 pipe what a product does: by integers where the
// result is a normal float
__device__ __forceinline__ float narrow(double x) {
    if (narrow_range(x)) return __uint_as_float(narrow_bits(x));
    float f;
    asm volatile("cvt.rn.f32.f64 %0, %1;" : "=f"(f) : "d"(x));
    return f;
}
__device__ __forceinline__ double widen(float f) {
    const uint32_t b = __float_as_uint(f);
    if (((b & 0x7fffffffu) - 0x00800000u) < 0x7f000000u) return widen_bits(b);
    double d;
    asm volatile("cvt.f64.f32 %0, %1;" : "=d"(d) : "f"(f));
    return d;
}

// Sums and products as fused multiply-adds of three registers.  The FP64 pipe
// takes 15.8 SM cycles for a dfma whose operands are three registers and 18.7
// for a dadd, a dmul or a dfma with a constant operand (measured, any number of
// warps).  a + b = fma(a, 1, b) and a b = fma(a, b, -0) hold bit for bit (the
// -0 leaves the sign of a zero product), provided the compiler cannot see the
// constants: they are read from memory into registers once per thread.
static __device__ double g_fma_one = 1.0, g_fma_nzero = -0.0;
struct Fma {
    double one, nzero;
    __device__ __forceinline__ Fma()
        : one(*(const volatile double*)&g_fma_one), nzero(*(const volatile double*)&g_fma_nzero) {}
    __device__ __forceinline__ double add(double a, double b) const { return fma(a, one, b); }
    __device__ __forceinline__ double mul(double a, double b) const { return fma(a, b, nzero); }
    // a / b, r = 1 / b to an ulp (the same r serves every dividend)
    __device__ __forceinline__ double quot(double a, double b, double r) const {
        double q;
        if (int_range_or_zero(a) && int_range(b) && int_range(r) && rn_div_int(a, b, r, q)) return q;
        return a / b;
    }
    // a b on the integer pipes where both are in their range
    __device__ __forceinline__ double prod(double a, double b) const {
        if (int_range_or_zero(a) && int_range_or_zero(b)) return rn_mul_int(a, b);
        return pipe_fma(a, b, nzero);
    }
};

// cw_exp (dcpse_common.cuh) bit for bit in 18 FP64 instructions of the short
// kind: the argument checks and the power of two on integers, the rounding to
// an integer by adding 1.5 2^52 (whose low bits are then k), the coefficients
// from shared memory (a constant operand is the slow kind).
struct ExpShared {
    double c[18];  // 1/13! .. 1/2!, then 1, INV_LN2, 1.5 2^52, LN2_HI, LN2_LO, unused
};
__device__ __forceinline__ void stage_exp(ExpShared& X) {
    const double c[18] = {0x1.6124613a86d09p-33, 0x1.1eed8eff8d898p-29, 0x1.ae64567f544e4p-26, 0x1.27e4fb7789f5cp-22,
                          0x1.71de3a556c734p-19, 0x1.a01a01a01a01ap-16, 0x1.a01a01a01a01ap-13, 0x1.6c16c16c16c17p-10,
                          0x1.1111111111111p-7,  0x1.5555555555555p-5,  0x1.5555555555555p-3,  0x1.0000000000000p-1,
                          1.0,                   0x1.71547652b82fep+0,  0x1.8p52,              0x1.62e42ff000000p-1,
                          -0x1.718432a1b0e26p-35, 0.0};
    if (threadIdx.x == 0)
        for (int i = 0; i < 18; ++i) X.c[i] = c[i];
}
__device__ __forceinline__ double cw_exp(const Fma& F, const ExpShared& X, double x) {
    if (((uint32_t)__double2hiint(x) & 0x7fffffffu) >= 0x4085e000u) return cw_exp(x);  // |x| >= 700, NaN
    const volatile double* c = X.c;
    const double magic = c[14];
    const double t = F.add(F.mul(x, c[13]), magic);
    const int k = __double2loint(t);
    const double kd = F.add(t, -magic);
    double r = fma(-kd, c[15], x);
    r = fma(-kd, c[16], r);
    const double one = c[12];
    double p = fma(c[0], r, c[1]);
#pragma unroll
    for (int i = 2; i < 12; ++i) p = fma(p, r, c[i]);
    p = fma(p, r, one);
    p = fma(p, r, one);
    // 0.7 < p < 1.5 and |k| <= 1010: p 2^k is normal
    return __hiloint2double(__double2hiint(p) + (int)((unsigned)k << 20), __double2loint(p));
}
#endif

}  // namespace dcpse
