// FP64 dot products in fixed point on the integer pipes.
//
// The FP64 unit issues 2 FMAs per clock per SM here; the 32-bit integer
// multiply-add with a 64-bit sum (IMAD.WIDE) about 56, on another pipe (a
// probe's rates at 1.92 GHz; both run side by side undisturbed).  A dot product
// of doubles over a common exponent is a dot product of integers: with
//
//     B_k = (bh 2^31 + bl) 2^-sb,  A_k = (ah 2^31 + al) 2^-(s + 31)
//
// the sums hh = sum ah bh and w = sum (ah bl + al bh), 64-bit and exact, give
// sum A B = (hh + w/2^31) 2^(31 - s - sb) up to the products al bl, below half a
// unit of hh: three IMAD.WIDE a term, and one rounding to FP64 at the end.
#pragma once

#include "common.cuh"

namespace b200 {

// The magnitude that the largest exponent is taken from
__device__ __forceinline__ int hi_abs(double x) { return __double2hiint(x) & 0x7fffffff; }

// Exponents that the fixed-point form does not take (near the ends of the
// range, infinities, NaNs; zeros it does take)
__device__ __forceinline__ bool out_of_range(int mx) {
    return mx != 0 && (unsigned)(mx - (128 << 20)) >= (unsigned)((1900 - 128) << 20);
}

// x as (bh 2^31 + bl) 2^-(1022 + BITS - emax), |bh| < 2^(BITS - 31), |bl| < 2^31,
// both of x's sign: with the mantissa's leading one at bit 63 of (vh, vl), bh is
// vh shifted down by 95 - 32 - BITS and the exponent difference d, bl the 31
// bits below.  In 32-bit operations throughout (a 64-bit shift by a variable
// issues as slowly as a quarter of these).
__device__ __forceinline__ unsigned shr_clamp(unsigned x, unsigned n) {
    return __funnelshift_rc(x, 0u, n);
}

// (down: emax + 63 - BITS)
__device__ __forceinline__ int2 split_down(double x, int down) {
    const int hi = __double2hiint(x), lo = __double2loint(x);
    // (zeros and subnormals: a difference of at least 64, so that nothing is
    // left of them)
    const int d = down - ((hi >> 20) & 0x7ff);
    const unsigned vh = __funnelshift_l(lo, (hi & 0xfffff) | 0x100000, 11), vl = (unsigned)lo << 11;
    int bh = (int)shr_clamp(vh, d);
    int bl = (int)(shr_clamp(__funnelshift_rc(vl, vh, d + 1), max(d - 31, 0)) & 0x7fffffffu);
    if (hi < 0) {
        bh = -bh;
        bl = -bl;
    }
    return make_int2(bh, bl);
}

template <int BITS>
__device__ __forceinline__ int2 split(double x, int emax) {
    return split_down(x, emax + 63 - BITS);
}

// t 2^sc rounded to FP64, |t| < 2^61, on the integer pipes: the conversion
// instruction runs on the FP64 unit, at its rate of 2 a clock and SM
__device__ __forceinline__ double fixed_to_f64(long long t, int sc) {
    const int sg = (int)(t >> 63);
    const unsigned long long mag = (unsigned long long)((t ^ (long long)sg) - (long long)sg);
    unsigned h = (unsigned)(mag >> 32), l = (unsigned)mag;
    int e = 1023 + 62 + sc;
    if (h == 0) {
        h = l;
        l = 0;
        e -= 32;
    }
    // The leading one to bit 63; its 53 bits rounded (a carry out of them lands
    // in the exponent, as it should)
    const int lz = __clz((int)h);
    const unsigned nh = __funnelshift_l(l, h, lz), nl = l << (lz & 31);
    const unsigned long long q =
        (((unsigned long long)nh << 32 | nl) >> 11) + ((nl >> 10) & 1u);
    const int hi = (int)(q >> 32) + (e - lz) * (1 << 20) + (sg & (int)0x80000000);
    return h == 0 ? 0.0 : __hiloint2double(hi, (int)q);
}

// The same with the conversion on the FP64 unit (kernels that leave it idle)
__device__ __forceinline__ double fixed_to_f64_cvt(long long t, int sc) {
    const double y = (double)t;
    return t == 0 ? 0.0 : __hiloint2double(__double2hiint(y) + sc * (1 << 20), __double2loint(y));
}

// Sums of products of one output
struct Fx {
    long long hh, w;
    __device__ __forceinline__ void clear() {
        hh = 0;
        w = 1ll << 30;
    }
    __device__ __forceinline__ void mad(int2 a, int2 b) {
        hh += (long long)a.x * b.x;
        w += (long long)a.x * b.y;
        w += (long long)a.y * b.x;
    }
    __device__ __forceinline__ long long total() const { return hh + (w >> 31); }
    // sc: emax - s - (991 + BITS)
    __device__ __forceinline__ double value(int sc) const { return fixed_to_f64(total(), sc); }
    __device__ __forceinline__ double value_cvt(int sc) const {
        return fixed_to_f64_cvt(total(), sc);
    }
};

}  // namespace b200
