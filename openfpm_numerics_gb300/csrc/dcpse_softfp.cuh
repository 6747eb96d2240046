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
#define DCPSE_HD __host__ __device__ __forceinline__
#else
#define DCPSE_HD inline
#endif

namespace dcpse {

DCPSE_HD uint64_t dbits(double x) {
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t u;
    std::memcpy(&u, &x, sizeof u);
    return u;
#endif
}

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
    return (((uint32_t)(dbits(x) >> 32) & 0x7fffffffu) - 0x30000000u) < 0x20000000u;
}
// ... or a zero, which products with such numbers may have on one side
DCPSE_HD bool int_range_or_zero(double x) { return int_range(x) || (dbits(x) << 1) == 0; }

// RN(a b), bit for bit IEEE round to nearest even, for a and b in int_range or
// zero.  The 106-bit product of the significands, its top 64 bits with a
// sticky bit, normalised by at most one place, rounded at bit 11; the implicit
// one of the result carries into the exponent field.
DCPSE_HD double rn_mul_int(double a, double b) {
    const uint64_t ab = dbits(a), bb = dbits(b);
    const uint32_t ah = (uint32_t)(ab >> 32), al = (uint32_t)ab, bh = (uint32_t)(bb >> 32), bl = (uint32_t)bb;
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

#if defined(__CUDACC__)
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
};
#endif

}  // namespace dcpse
