// selftest.cu -- compares, on the GPU the library runs on, the truncation of the
// Student-t variance sums (exact_arith.cuh) with the conversion it replaces, the
// reciprocal and division of pair_math.cuh with the compiler's, and the fixed-point
// sums of fx.cuh with 128-bit integers.
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/recon_track.h"
#include "exact_arith.cuh"
#include "fx.cuh"
#include "pair_math.cuh"

namespace rt {

void set_last_error(const char *msg);

namespace {

__device__ __forceinline__ void add_count(unsigned long long *dst, unsigned long long c) {
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(dst, c);
}

// every float x in [0, 2^23): trunc_small(x) against (int)x
__global__ void k_check_trunc(unsigned long long *bad) {
    unsigned long long c = 0;
    uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < 0x4B000000u; b += stride) {
        float x = __uint_as_float(b);
        c += trunc_small(x) != (int)x;
    }
    add_count(bad, c);
}

// every mantissa in seven binades of [2^-60, 2^60], the first and the last among
// them, and 2^60, both signs: the reciprocal against the correctly rounded one
__global__ void k_check_rcp(unsigned long long *bad) {
    unsigned long long c = 0;
    uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t m = blockIdx.x * blockDim.x + threadIdx.x; m < 0x800000u; m += stride)
        for (uint32_t k = 0; k < 8; k++) {
            uint32_t E = k < 6 ? 127 - 60 + 20 * k : 127 + 53 + k;  // 67, 87, .. 167, 186, 187
            if (k == 7 && m) continue;
            for (uint32_t sign = 0; sign < 2; sign++) {
                float b = __uint_as_float(sign << 31 | E << 23 | m), y = __frcp_rn(b);
                float2 y2 = rcp_rn2(dup2(b));
                c += rcp_rn(b) != y || y2.x != y || y2.y != y;
            }
        }
    add_count(bad, c);
}

// a linear congruential sequence a thread
struct Draws {
    unsigned long long s;
    __device__ __forceinline__ explicit Draws(unsigned long long seed)
        : s((blockIdx.x * blockDim.x + threadIdx.x) * 0x9E3779B97F4A7C15ull + seed) {}
    __device__ __forceinline__ uint32_t bits() {
        s = s * 6364136223846793005ull + 1442695040888963407ull;
        return (uint32_t)(s >> 32);
    }
    // a value of either sign in [2^lo, 2^hi]
    __device__ __forceinline__ float value(int lo, int hi) {
        uint32_t m = bits(), E = 127 + lo + (bits() >> 8) % (hi - lo + 1);
        return __uint_as_float((m & 0x80000000u) | E << 23 | (E == 127u + hi ? 0u : m & 0x7fffffu));
    }
};

// pseudo-random operands of the range: quotients against the compiler's division,
// and packed sums and differences of products against separately rounded ones
__global__ void k_check_div(unsigned long long *bad, int per_thread) {
    unsigned long long c = 0;
    Draws draw(12345);
    for (int i = 0; i < per_thread; i++) {
        float a0 = draw.value(-60, 60), a1 = draw.value(-60, 60), b = draw.value(-60, 60);
        float2 q = div_rn2(make_float2(a0, a1), dup2(-b), rcp_rn2(dup2(b)));
        // a product and a sum stay two roundings
        float2 s2 = add2(mul2(make_float2(a0, a1), dup2(b)), make_float2(a1, a0), unseen_one());
        float2 d2 = sub2(make_float2(a1, a0), mul2(make_float2(a0, a1), dup2(b)));
        c += s2.x != __fadd_rn(__fmul_rn(a0, b), a1) || s2.y != __fadd_rn(__fmul_rn(a1, b), a0);
        c += d2.x != __fsub_rn(a1, __fmul_rn(a0, b)) || d2.y != __fsub_rn(a0, __fmul_rn(a1, b));
        c += !div_in_range(a0, a1, b) || div_rn(a0, -b, rcp_rn(b)) != a0 / b || q.x != a0 / b || q.y != a1 / b;
    }
    add_count(bad, c);
}

// Numerators below the range, which some callers pass without a look: zeros,
// denormal and small values, in the callers' own expressions, and as a quotient
// (IcpTaps), which is exact down to numerators of 2^-102 and below that within a
// unit in the last place.
__global__ void k_check_small(unsigned long long *bad, int per_thread) {
    unsigned long long c = 0;
    Draws draw(54321);
    auto over = [](float a, float b) { return div_rn2(dup2(a), dup2(-b), rcp_rn2(dup2(b))); };
    for (int i = 0; i < per_thread; i++) {
        uint32_t r = draw.bits();
        // exponent field 0 .. 66, a zero now and then
        float tiny = (r & 63u) == 0 ? 0.0f : __uint_as_float((r >> 8 & 0x7fffffu) | (draw.bits() >> 8) % 67 << 23);
        float sigma2 = fabsf(draw.value(-20, 60)), scale = fabsf(draw.value(-7, 1)), f = fabsf(draw.value(-20, 20));
        // Student-t: 5 + r^2 / sigma^2, by either form
        float t = 5.0f + tiny / sigma2;
        float2 q = over(tiny, sigma2);
        c += 5.0f + div_rn(tiny, -sigma2, rcp_rn(sigma2)) != t || 5.0f + q.x != t || 5.0f + q.y != t;
        // Tukey: 1 - (|r| / scale / 4.6851)^2
        float2 u = over(tiny, scale), ub = div_rn2(u, dup2(-4.6851f), dup2(1.0f / 4.6851f));
        float v = tiny / scale / 4.6851f;
        c += 1.0f - ub.x * ub.x != 1.0f - v * v || !(u.x <= 4.6851f);
        // depth: 1 - e / 1e4
        float2 e = div_rn2(dup2(tiny), dup2(-10000.0f), dup2(1.0f / 10000.0f));
        c += 1.0f - e.x != 1.0f - tiny / 10000.0f;
        // a coordinate over a focal length
        float a = r & 64u ? -tiny : tiny, exact = a / f;
        float2 p = over(a, f);
        c += fabsf(a) >= 0x1p-102f ? p.x != exact : !(fabsf(p.x - exact) <= 0x1p-23f * fabsf(exact) + 0x1p-126f);
    }
    add_count(bad, c);
}

// a sum in units of 2^-64, rounded to FP64: to 64 bits of which the last is set
// when any bit after it was, then by the hardware's conversion
__device__ double round_q64(unsigned __int128 q) {
    bool neg = (q >> 127) != 0;
    unsigned __int128 u = neg ? (unsigned __int128)0 - q : q;
    int s = 0;
    for (; (u >> s >> 64) != 0; s++) {}
    unsigned long long top = (unsigned long long)(u >> s);
    if ((u & (((unsigned __int128)1 << s) - 1)) != 0) top |= 1ull;
    double v = ldexp(__ull2double_rn(top), s - 64);
    return neg ? -v : v;
}
__device__ __forceinline__ bool same(double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b); }

// One value of every exponent and sign (mantissas of all zeros, all ones and
// random bits), and sums of 40: fx_accumulate against fx_split and against the
// value in 128 bits, and what is out of range.
__global__ void k_check_fx_sum(unsigned long long *bad, int per_thread) {
    unsigned long long c = 0;
    Draws draw(777);
    for (int i = 0; i < per_thread; i++) {
        uint32_t acc[4] = {0u, 0u, 0u, 0u};
        unsigned __int128 want = 0;
        long long limbs[kFxLimbs] = {0, 0, 0, 0};
        int n = i & 1 ? 40 : 1, flag = 0, split_flag = 0;
        bool out = false;
        for (int k = 0; k < n; k++) {
            uint32_t r = draw.bits(), E = n > 1 ? (draw.bits() >> 8) % 175u : (draw.bits() >> 8) % 256u;
            uint32_t M = draw.bits() & 0x7fffffu;
            if ((r & 3u) < 2u) M = r & 1u ? 0x7fffffu : 0u;
            float v = __uint_as_float((r & 0x80000000u) | E << 23 | M);
            fx_accumulate(acc, v, flag);
            int k0;
            long long lo, hi;
            fx_split(v, k0, lo, hi, split_flag);
            limbs[k0] += lo;
            if (hi) limbs[k0 + 1] += hi;
            if (E >= 175u) {
                out = true;
                continue;
            }
            // (a denormal value is below the unit)
            unsigned __int128 m = E ? (unsigned __int128)(M | 0x800000u) : 0;
            int s = (int)E - 86;
            m = s >= 0 ? m << s : (s <= -24 ? 0 : m >> -s);
            want += r >> 31 ? (unsigned __int128)0 - m : m;
        }
        unsigned __int128 got = (unsigned __int128)acc[3] << 96 | (unsigned __int128)acc[2] << 64 |
                                (unsigned __int128)acc[1] << 32 | acc[0];
        c += got != want || (flag != 0) != out || (split_flag != 0) != out;
        c += !same(fx_to_double(limbs), round_q64(want));
    }
    add_count(bad, c);
}

// fx_to_double of limbs that overlap, of sums of every length, and of halves: a
// 53-bit mantissa (random, even, odd, all ones) with one half of its last place
// after it, and a little more or less than that
__global__ void k_check_fx_round(unsigned long long *bad, int per_thread) {
    unsigned long long c = 0;
    Draws draw(4242);
    for (int i = 0; i < per_thread; i++) {
        unsigned long long a = (unsigned long long)draw.bits() << 32 | draw.bits();
        unsigned long long b = (unsigned long long)draw.bits() << 32 | draw.bits();
        uint32_t r = draw.bits();
        unsigned __int128 q;
        if (r & 1u) {
            unsigned long long m = (r & 6u) == 6u ? (1ull << 53) - 1 : a >> 11 | 1ull << 52;
            int s = (r >> 8) % 73u;  // the half's place
            q = ((unsigned __int128)m << 1 | 1) << s;
            if (s && (r & 24u) == 8u) q += 1;
            if ((r & 24u) == 16u) q -= 1;
        } else {
            q = ((unsigned __int128)a << 64 | b) >> (1 + (r >> 8) % 127u);
        }
        if (r & 32u) q = (unsigned __int128)0 - q;
        long long limbs[kFxLimbs];
        for (int k = 0; k < kFxLimbs; k++) limbs[k] = (long long)(uint32_t)(q >> (32 * k));
        limbs[3] = (int)(uint32_t)limbs[3];
        c += !same(fx_to_double(limbs), round_q64(q));
        // the same total with pieces moved from limb to limb
        for (int k = 0; k < kFxLimbs - 1; k++) {
            long long t = (int)draw.bits() >> 4;
            limbs[k] += t * (1ll << 32);
            limbs[k + 1] -= t;
        }
        c += !same(fx_to_double(limbs), round_q64(q));
    }
    add_count(bad, c);
}

}  // namespace
}  // namespace rt

namespace {

// runs `launch` on a zeroed counter and returns the count
template <class Launch> int count_mismatches(int64_t *mismatches, const char *name, Launch launch) {
    if (!mismatches) {
        rt::set_last_error(name);
        return RECON_ERR_INVALID_ARG;
    }
    unsigned long long *d = nullptr;
    cudaError_t e = cudaMalloc(&d, sizeof(unsigned long long));
    if (e == cudaSuccess) e = cudaMemset(d, 0, sizeof(unsigned long long));
    if (e == cudaSuccess) {
        launch(d);
        e = cudaGetLastError();
    }
    unsigned long long h = 0;
    if (e == cudaSuccess) e = cudaMemcpy(&h, d, sizeof(h), cudaMemcpyDeviceToHost);
    if (d) cudaFree(d);
    if (e != cudaSuccess) {
        rt::set_last_error(cudaGetErrorString(e));
        return RECON_ERR_CUDA;
    }
    *mismatches = (int64_t)h;
    return RECON_OK;
}

}  // namespace

extern "C" int recon_selftest_exact_arith(int64_t *mismatches) {
    return count_mismatches(mismatches, "recon_selftest_exact_arith: null argument",
                            [](unsigned long long *d) { rt::k_check_trunc<<<152 * 8, 256>>>(d); });
}

extern "C" int recon_selftest_division(int64_t *mismatches) {
    return count_mismatches(mismatches, "recon_selftest_division: null argument", [](unsigned long long *d) {
        rt::k_check_rcp<<<152 * 8, 256>>>(d);
        rt::k_check_div<<<152 * 8, 256>>>(d, 4000);
        rt::k_check_small<<<152 * 8, 256>>>(d, 1000);
    });
}

extern "C" int recon_selftest_fixed_point(int64_t *mismatches) {
    return count_mismatches(mismatches, "recon_selftest_fixed_point: null argument", [](unsigned long long *d) {
        rt::k_check_fx_sum<<<152 * 4, 256>>>(d, 200);
        rt::k_check_fx_round<<<152 * 4, 256>>>(d, 400);
    });
}
