// FP64 interpolation sums in 64-bit fixed point.
//
// A tricubic row is 84 multiply-adds, and this GPU does 1.7 FP64 operations a
// clock and SM (DFMA, DADD and DMUL alike, measured) against 60 integer
// 32 x 32 + 64 -> 64 multiply-adds.  So the E sums of FP64 vectors are block
// floating point: the 64 values of a stencil are aligned to the stencil's
// largest exponent e as integers of 61 bits and a sign, the 1-D weights are
// integers w 2^62, and a product keeps its 64 high bits from three multiply-adds
// of 32-bit halves (the product of the low halves is below the last bit).
// Each of the three 1-D sums scales by 2^62 / 2^64, so a row ends as an integer
// of 2^(e - 54): 2^-55 of the largest value, rounded to nearest there and once
// more to 53 bits.  Plain FP64 rounds 84 times at 2^-53 of the running sums;
// measured against 64-bit-exact rows the error here is the smaller one
// (k_epass1, k_epass32x).
//
// A stencil with an infinity, a NaN or only values below 2^-895 (nothing is
// left of the exponent range to align to) takes the FP64 sum instead.
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
// (at least this value's own), truncated.  Zeros and subnormals come out as 0
// or -1 (e is at least 128 above them).
__device__ __forceinline__ Fx fx_from_double(uint32_t hi, uint32_t lo, uint32_t e20) {
    const uint32_t d = min((e20 - (hi & FX_EXP)) >> 20, 63u);
    const uint32_t mh = (hi & 0xfffffu) | 0x100000u;
    const uint64_t m = ((uint64_t)__funnelshift_l(lo, mh, 8) << 32) | (uint64_t)(lo << 8);
    const uint64_t v = m >> d;
    const uint32_t s = (uint32_t)((int)hi >> 31);  // ones' complement of a negative value: one unit off
    return fx_split((int64_t)((((uint64_t)((uint32_t)(v >> 32) ^ s)) << 32) | (uint64_t)((uint32_t)v ^ s)));
}

// the double v in units of 2^(e - 59), 60 bits: six of them add up without overflow
__device__ __forceinline__ int64_t fx60_from_double(double v, uint32_t e20) {
    const uint32_t hi = (uint32_t)__double2hiint(v), lo = (uint32_t)__double2loint(v);
    const uint32_t d = min((e20 - (hi & FX_EXP)) >> 20, 63u);
    const uint32_t mh = (hi & 0xfffffu) | 0x100000u;
    const uint64_t m = ((uint64_t)__funnelshift_l(lo, mh, 7) << 32) | (uint64_t)(lo << 7);
    const uint64_t r = m >> d;
    const uint32_t s = (uint32_t)((int)hi >> 31);
    return (int64_t)((((uint64_t)((uint32_t)(r >> 32) ^ s)) << 32) | (uint64_t)((uint32_t)r ^ s));
}

// a b + c on 32-bit signed factors
__device__ __forceinline__ int64_t fx_mad(int a, int b, int64_t c) {
    int64_t d;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
    return d;
}
// (sum_k x_k w_k) / 2^64, rounded
__device__ __forceinline__ int64_t fx_dot4(const Fx (&x)[4], const Fx (&w)[4]) {
    int64_t c = 0x80000000ll;
#pragma unroll
    for (int k = 0; k < 4; ++k) c = fx_mad(x[k].l, w[k].h, fx_mad(x[k].h, w[k].l, c));
    int64_t a = c >> 32;
#pragma unroll
    for (int k = 0; k < 4; ++k) a = fx_mad(x[k].h, w[k].h, a);
    return a;
}
// the same sum term by term
struct FxSum {
    int64_t c = 0x80000000ll, a = 0;
    __device__ __forceinline__ void add(Fx x, Fx w) {
        c = fx_mad(x.l, w.h, fx_mad(x.h, w.l, c));
        a = fx_mad(x.h, w.h, a);
    }
    __device__ __forceinline__ int64_t get() const { return a + (c >> 32); }
};

// the row sum r 2^(e - 54) as a double
__device__ __forceinline__ double fx_to_double(int64_t r, uint32_t e20) {
    return (double)r * __hiloint2double((int)(e20 - (54u << 20)), 0);
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
