// The FP64 product rounded to nearest even, formed on the integer pipe.
//
// On sm_103a the FP64 pipe issues 1.68 lane operations per cycle and SM, whatever the operation;
// the integer pipe does this product at 2.27 per cycle and SM beside it (both measured; one of
// each in turn runs at the FP64 pipe's rate).  A kernel that is bound by the FP64 pipe sheds the
// multiplications it hands over.
//
// Significands as 53-bit integers, b's shifted up by 11 so that the product's upper 64 bits hold
// the result's 53 or 52 bits and the lower 64 the rest; one bit of normalisation, then the
// rounding increment from the rest (sticky) and the last bit, carried into the exponent.
// Exact for zeros and for operands whose exponents lie in [-255, 256]; for any other operand
// (subnormal, near the ends of the range, infinite, not a number) `bad` becomes nonzero and the
// result is not meaningful: the caller multiplies again in floating point.
#pragma once
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define DUGKS_HD __host__ __device__ __forceinline__
#else
#define DUGKS_HD inline
#endif

namespace dugks {

DUGKS_HD uint32_t shl_from(uint32_t lo, uint32_t hi, uint32_t n) {  // upper word of (hi:lo) << n, n < 32
#ifdef __CUDA_ARCH__
    return __funnelshift_l(lo, hi, n);
#else
    return (uint32_t)(((((uint64_t)hi << 32) | lo) << n) >> 32);
#endif
}
DUGKS_HD void words_of(double d, uint32_t &hi, uint32_t &lo) {
#ifdef __CUDA_ARCH__
    hi = (uint32_t)__double2hiint(d);
    lo = (uint32_t)__double2loint(d);
#else
    uint64_t v;
    std::memcpy(&v, &d, 8);
    hi = (uint32_t)(v >> 32);
    lo = (uint32_t)v;
#endif
}
DUGKS_HD double double_of(uint32_t hi, uint32_t lo) {
#ifdef __CUDA_ARCH__
    return __hiloint2double((int)hi, (int)lo);
#else
    const uint64_t v = ((uint64_t)hi << 32) | lo;
    double d;
    std::memcpy(&d, &v, 8);
    return d;
#endif
}

DUGKS_HD double mul_int(double a, double b, uint32_t &bad) {
    uint32_t ah, al, bh, bl;
    words_of(a, ah, al);
    words_of(b, bh, bl);
    const uint32_t ta = ah & 0x7ff00000u, tb = bh & 0x7ff00000u;
    const bool za = ((ah + ah) | al) == 0, zb = ((bh + bh) | bl) == 0;
    bad |= ((za ? 0u : ta - 0x30000000u) | (zb ? 0u : tb - 0x30000000u)) & 0xE0000000u;
    const uint32_t a1 = (ah & 0xfffffu) | 0x100000u, bm = (bh & 0xfffffu) | 0x100000u;
    const uint32_t b1 = shl_from(bl, bm, 11), b0 = bl << 11;
    const uint64_t p0 = (uint64_t)al * b0;
    const uint64_t p1 = (uint64_t)a1 * b0 + (p0 >> 32);
    const uint64_t p2 = (uint64_t)al * b1 + (uint32_t)p1;
    const uint64_t H = (uint64_t)a1 * b1 + (p1 >> 32) + (p2 >> 32);
    uint32_t hh = (uint32_t)(H >> 32), hl = (uint32_t)H, lh = (uint32_t)p2, ll = (uint32_t)p0;
    const uint32_t nb = ~hh & 0x100000u, n = nb >> 20;  // one place up where bit 52 is clear
    hh = shl_from(hl, hh, n);
    hl = shl_from(lh, hl, n);
    lh = shl_from(ll, lh, n);
    ll <<= n;
    const uint32_t rest = lh | (ll != 0 ? 1u : 0u);
    const uint64_t r = (((uint64_t)hh << 32) | hl) + (((uint64_t)rest + (hl & 1u) + 0x7fffffffu) >> 32);
    const uint32_t hi = (uint32_t)(r >> 32) + ta + tb - 0x3ff00000u - nb, sign = (ah ^ bh) & 0x80000000u;
    return za || zb ? double_of(sign, 0) : double_of(hi | sign, (uint32_t)r);
}

}  // namespace dugks
