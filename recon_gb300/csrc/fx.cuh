// fx.cuh -- exact fixed-point accumulation of FP32 values on the GPU.
//
// A value is the integer sum_k L[k] * 2^(32k) in units of 2^-64, held as four
// 64-bit limb sums.  An FP32 input is truncated toward zero at 2^-64 and splits
// into at most two adjacent 32-bit pieces, so limb sums never carry and can be
// added with plain integer atomics in any order: the total is the exact sum of
// the inputs.  It is rounded once to FP64 (nearest, ties to even) with integer
// arithmetic only.  Inputs must satisfy |v| < 2^48; Inf, NaN and larger values
// set a flag instead.  The oracle's orc_fx_add / orc_fx_to_double are the same
// definition.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "track_kernels.cuh"

namespace rt {

// v -> (limb index k0, piece for limb k0, piece for limb k0+1); sets bad when
// v is out of range.  Zero pieces mean nothing to add.
__device__ __forceinline__ void fx_split(float v, int &k0, long long &lo, long long &hi, int &bad) {
    uint32_t bits = __float_as_uint(v);
    uint32_t E = (bits >> 23) & 0xffu, M = bits & 0x7fffffu;
    k0 = 0;
    lo = 0;
    hi = 0;
    if (E == 0xffu) { bad = 1; return; }
    uint64_t m = (E == 0) ? (uint64_t)M : (uint64_t)(M | 0x800000u);
    int e = (E == 0) ? -149 : (int)E - 150;
    if (m == 0) return;
    if (e >= 25) { bad = 1; return; }
    int s = e + 64;
    if (s < 0) {
        m = (-s >= 24) ? 0 : (m >> -s);
        s = 0;
    }
    uint64_t t = m << (s & 31);
    k0 = s >> 5;
    lo = (long long)(t & 0xffffffffu);
    hi = (long long)(t >> 32);
    if (bits >> 31) { lo = -lo; hi = -hi; }
}

// Adds v to a 128-bit sum of the same units held as four 32-bit words (two's
// complement), in registers; sets bad when v is out of range.
__device__ __forceinline__ void fx_accumulate(uint32_t *a, float v, int &bad) {
    uint32_t bits = __float_as_uint(v), E = (bits >> 23) & 0xffu;
    if (E >= 175u) {  // |v| >= 2^48, Inf or NaN
        bad = 1;
        return;
    }
    // below 2^-64 the value is cut to units of 2^-64 (E == 0 shifts everything out)
    uint32_t m = (bits & 0x7fffffu) | 0x800000u;
    int s = (int)E - 86;
    if (s < 0) {
        m = s <= -24 ? 0u : m >> -s;
        s = 0;
    }
    uint64_t t = (uint64_t)m << (s & 31);
    uint32_t lo = (uint32_t)t, hi = (uint32_t)(t >> 32), neg = bits >> 31, sign = 0u - neg;
    int k = s >> 5;  // 0..2
    uint32_t w0 = (k == 0 ? lo : 0u) ^ sign, w1 = (k == 0 ? hi : (k == 1 ? lo : 0u)) ^ sign;
    uint32_t w2 = (k == 1 ? hi : (k == 2 ? lo : 0u)) ^ sign, w3 = (k == 2 ? hi : 0u) ^ sign;
    asm("{\n.reg .u32 c;\nadd.cc.u32 c, %8, %9;\naddc.cc.u32 %0, %0, %4;\naddc.cc.u32 %1, %1, %5;\n"
        "addc.cc.u32 %2, %2, %6;\naddc.u32 %3, %3, %7;\n}\n"
        : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3])
        : "r"(w0), "r"(w1), "r"(w2), "r"(w3), "r"(sign), "r"(neg));
}

__device__ __forceinline__ double fx_to_double(const long long *L) {
    // the sum modulo 2^128, limb by limb, and its magnitude
    static_assert(kFxLimbs == 4, "a 128-bit sum");
    long long c = L[0];
    unsigned long long lo = (uint32_t)c;
    c = (c >> 32) + L[1];
    lo |= (unsigned long long)c << 32;
    c = (c >> 32) + L[2];
    unsigned long long hi = (uint32_t)c;
    c = (c >> 32) + L[3];
    hi |= (unsigned long long)c << 32;
    unsigned long long sign = hi & (1ull << 63);
    if (sign) {
        lo = 0ull - lo;
        hi = ~hi + (lo == 0);
    }
    if ((hi | lo) == 0) return 0.0;
    // its first one to the top bit; 53 bits are the mantissa, the others round it
    int lead = hi ? __clzll((long long)hi) : 64 + __clzll((long long)lo), s = lead & 63;
    if (lead >= 64) {
        hi = lo;
        lo = 0;
    }
    if (s) {
        hi = hi << s | lo >> (64 - s);
        lo <<= s;
    }
    unsigned long long mant = hi >> 11;
    uint32_t rest = (uint32_t)hi & 0x7ffu;
    mant += rest > 0x400u || (rest == 0x400u && (lo != 0 || (mant & 1)));
    // (a mantissa that rounding takes to 2^53 carries into the exponent)
    return __longlong_as_double(
        (long long)(sign | (((unsigned long long)(1023 + 63 - lead) << 52) + (mant - (1ull << 52)))));
}

}  // namespace rt
