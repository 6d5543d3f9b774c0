// FP64 interpolation sums in 64-bit fixed point.
//
// A tricubic row is 84 multiply-adds, and this GPU does 1.7 FP64 operations a
// clock and SM (DFMA, DADD and DMUL alike, measured) against 60 integer
// 32 x 32 + 64 -> 64 multiply-adds.  So the E sums of FP64 vectors are block
// floating point: the 64 values of a stencil are aligned to the stencil's
// largest exponent e as integers of 61 bits and a sign, the 1-D weights are
// integers w 2^62, and a product keeps its high bits from three multiply-adds
// of 32-bit halves (the product of the low halves is below the last bit).
// All three 1-D sums are kept in units of 2^(e - 60), two bits more than the high
// word of the product, and stay within 62 bits: a cubic row's weights sum to at
// most 1.25 in magnitude an axis.
//
// So a row is off by at most 25 units of 2^(e - 60), usually by half of one, and
// once more by its conversion to 53 bits, where the FP64 sum rounds up to 12 times
// at 2^-53 of the row's own terms.  It is the fixed-point sum only where that is
// the better one: a row whose terms sum |w x| is not seen to reach 2^(e - 7) (from
// its value, fx_small, else from its eight central terms, fx_weak) takes the FP64
// sum.  These are rows that hardly weigh their largest value: a closest point next
// to a grid node of small value, the steep front of a decaying field.  Host
// restatements of 40 thousand rows a field, in units of 2^-53 sum |w x|, rms /
// largest error:
//   field                       FP64 sum     fixed point   rows redone
//   noise                       0.57 / 3.5   0.21 / 1.0    none
//   linear through zero         0.59 / 3.0   0.23 / 0.8    none
//   the same, 7 of 10 points by
//   a grid plane an axis        0.96 / 5.6   0.37 / 2.8    4e-3
//   exp(-d/dx)                  0.59 / 3.8   0.24 / 1.0    none
//   exp(-d/(0.3 dx))            0.32 / 2.4   0.30 / 2.4    0.84
//   a factor 1e-4 a cell        0.62 / 3.8   0.61 / 3.8    0.98
// Without that choice the last two rows are off by up to 470 and 4e6 such units.
// In solves 0.5 to 2 % of the rows take it, at the front of the first iterates; the
// choice costs 4 % of a solve and the rows redone 4 to 12 % (FP64, one vector at dx
// 0.025 on the sphere 16.0 -> 17.6 ms, 32 on the torus at 0.04 82.7 -> 96.9 ms).
//
// A stencil with an infinity, a NaN or only values below 2^-895 (nothing is
// left of the exponent range to align to) takes the FP64 sum as well.
//
// E(-x) is -E(x) bit for bit, as in FP64, although truncation and rounding are not
// symmetric here: a stencil is summed with the sign that makes one of its values
// positive (flip: its centre, or the first that is not zero).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace cpm {

// h 2^32 + l with a signed low half (a borrow is in h), so that both halves
// are operands of the signed 32-bit multiply
struct Fx {
    int h, l;
};

constexpr uint32_t FX_EXP = 0x7ff00000u;      // exponent field of a double's high word
constexpr uint32_t FX_EMIN = 128u << 20;      // smallest exponent field that is aligned to
constexpr double FX_WSCALE = 4611686018427387904.0;  // 2^62

__device__ __forceinline__ Fx fx_split(int64_t v) {
    Fx r;
    r.l = (int)(uint32_t)v;
    r.h = (int)(v >> 32) - (r.l >> 31);
    return r;
}

// the double (hi, lo) in units of 2^(e - 60), e the exponent of the field e20
// (at least this value's own), truncated; negated where the high bit of flip is
// set.  Zeros and subnormals come out as 0 or -1 (e is at least 128 above them).
__device__ __forceinline__ Fx fx_from_double(uint32_t hi, uint32_t lo, uint32_t e20, uint32_t flip) {
    const uint32_t d = min((e20 - (hi & FX_EXP)) >> 20, 63u);
    const uint32_t mh = (hi & 0xfffffu) | 0x100000u;
    const uint64_t m = ((uint64_t)__funnelshift_l(lo, mh, 8) << 32) | (uint64_t)(lo << 8);
    const uint64_t v = m >> d;
    const uint32_t s = (uint32_t)((int)(hi ^ flip) >> 31);  // ones' complement of a negative value: one unit off
    return fx_split((int64_t)((((uint64_t)((uint32_t)(v >> 32) ^ s)) << 32) | (uint64_t)((uint32_t)v ^ s)));
}

// the double v in units of 2^(e - 59), 60 bits: six of them add up without overflow.
// Ones' complement of a negative value: the caller counts them (sign: 0 or -1).
__device__ __forceinline__ int64_t fx60_from_double(double v, uint32_t e20, int &sign) {
    const uint32_t hi = (uint32_t)__double2hiint(v), lo = (uint32_t)__double2loint(v);
    const uint32_t d = min((e20 - (hi & FX_EXP)) >> 20, 63u);
    const uint32_t mh = (hi & 0xfffffu) | 0x100000u;
    const uint64_t m = ((uint64_t)__funnelshift_l(lo, mh, 7) << 32) | (uint64_t)(lo << 7);
    const uint64_t r = m >> d;
    const uint32_t s = (uint32_t)((int)hi >> 31);
    sign = (int)s;
    return (int64_t)((((uint64_t)((uint32_t)(r >> 32) ^ s)) << 32) | (uint64_t)((uint32_t)r ^ s));
}

// a b + c on 32-bit signed factors
__device__ __forceinline__ int64_t fx_mad(int a, int b, int64_t c) {
    int64_t d;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
    return d;
}
// (sum_k x_k w_k) / 2^62, rounded
__device__ __forceinline__ int64_t fx_dot4(const Fx (&x)[4], const Fx (&w)[4]) {
    int64_t c = 0x80000000ll >> 2, a = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        c = fx_mad(x[k].l, w[k].h, fx_mad(x[k].h, w[k].l, c));
        a = fx_mad(x[k].h, w[k].h, a);
    }
    return (a << 2) + (c >> 30);
}
// two terms of the last sum / 2^62, rounded: halves, because the small products of
// all four terms could pass 2^63
struct FxHalf {
    int64_t c = 0x80000000ll >> 2, a = 0;
    __device__ __forceinline__ void add(Fx x, Fx w) {
        c = fx_mad(x.l, w.h, fx_mad(x.h, w.l, c));
        a = fx_mad(x.h, w.h, a);
    }
    __device__ __forceinline__ int64_t get() const { return (a << 2) + (c >> 30); }
};

// a row sum r 2^(e - 60) below 2^(e - 7)
__device__ __forceinline__ bool fx_small(int64_t r) { return abs((int)(r >> 32)) < 1 << 21; }
// |x| |w| in units of 2^(u + 2), x.h in units of 2^u (w.h: 2^-30)
__device__ __forceinline__ uint32_t fx_abs_mul(uint32_t x, Fx w) { return __umulhi(x, (uint32_t)abs(w.h)); }
// the sum of a row's central |w x| of one plane, in units of 2^(e - 22), from its four values
__device__ __forceinline__ uint32_t fx_central(Fx x11, Fx x12, Fx x21, Fx x22, Fx wx, Fx wy1, Fx wy2, Fx wz1, Fx wz2) {
    const uint32_t y1 = fx_abs_mul((uint32_t)abs(x11.h), wz1) + fx_abs_mul((uint32_t)abs(x12.h), wz2);
    const uint32_t y2 = fx_abs_mul((uint32_t)abs(x21.h), wz1) + fx_abs_mul((uint32_t)abs(x22.h), wz2);
    return fx_abs_mul(fx_abs_mul(y1, wy1) + fx_abs_mul(y2, wy2), wx);
}
// both planes' below 2^(e - 7)
__device__ __forceinline__ bool fx_weak(uint32_t central) { return central < 1u << 15; }

// the row sum r 2^(e - 60) as a double, negated where the high bit of e20 is set
__device__ __forceinline__ double fx_to_double(int64_t r, uint32_t e20) {
    return (double)r * __hiloint2double((int)(e20 - (60u << 20)), 0);
}

// four consecutive weights
__device__ __forceinline__ void fx_load4(const int2 *w, Fx (&o)[4]) {
    const int4 a = __ldg((const int4 *)w), b = __ldg((const int4 *)w + 1);
    o[0] = Fx{a.y, a.x};
    o[1] = Fx{a.w, a.z};
    o[2] = Fx{b.y, b.x};
    o[3] = Fx{b.w, b.z};
}

// the same from shared memory
__device__ __forceinline__ void fx_lds4(const int2 *w, Fx (&o)[4]) {
    const int4 a = *(const int4 *)w, b = *((const int4 *)w + 1);
    o[0] = Fx{a.y, a.x};
    o[1] = Fx{a.w, a.z};
    o[2] = Fx{b.y, b.x};
    o[3] = Fx{b.w, b.z};
}

__device__ __forceinline__ Fx fx_lds1(const int2 *w) { return Fx{w->y, w->x}; }

// a weight as (l, h)
__host__ __device__ __forceinline__ int2 fx_weight(double w) {
    const int64_t v = (int64_t)rint(w * FX_WSCALE);
    const int l = (int)(uint32_t)v;
    return make_int2(l, (int)(v >> 32) - (l >> 31));
}

}  // namespace cpm
