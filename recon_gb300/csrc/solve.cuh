// solve.cuh -- FP64 6x6 solve and SE(3) pose update, executed by one warp.
//
// Every matrix element goes through the same sequence of FP64 operations as the
// oracle's restatement (orc_solve_cholesky, orc_expm_update), so the results
// are bit-identical; lanes only evaluate independent elements concurrently.
// On GB300 an FP64 warp instruction occupies its SM sub-partition for about 64
// cycles whether or not it depends on the previous one, and a divide or square
// root costs about ten of them.  The layout below therefore keeps the serial
// FP64 chain short: every product added to a sum is one fused multiply-add
// (the oracle's fma, one rounding), one reciprocal per pivot instead of a
// divide per element, lane-parallel substitutions, and comparisons of
// magnitudes on the integer bit patterns instead of FP64 compares.
#pragma once
#include <cuda_runtime.h>
#include <math.h>

namespace rt {

constexpr unsigned kFull = 0xffffffffu;

struct SolveScratch {
    double A[36], b[6];
    double tw[14];    // a small twist's entries: x, -x, 0
    double M[6][16];  // X, X2, X4, X6 / U0, V / N, D
    double E[16], T[16], Tinc[16];
    double lu_inv[3];
    int status;
};

// Pade (6,6) coefficients c_k = c_{k-1} (q-k+1) / (k (2q-k+1)), q = 6, in the
// oracle's FP64 evaluation order.
__device__ __constant__ const double kPade[7] = {0x1.0000000000000p+0, 0x1.0000000000000p-1, 0x1.d1745d1745d17p-4,
                                                 0x1.f07c1f07c1f07p-7, 0x1.4afd6a052bf5ap-10, 0x1.08cabb37565e2p-14,
                                                 0x1.937e11175f095p-20};

// |v| as an integer: for non-NaN values its order is the order of |v|
__device__ __forceinline__ long long abs_bits(double v) { return __double_as_longlong(v) & 0x7fffffffffffffffLL; }
constexpr long long kInfBits = 0x7ff0000000000000LL;

// 4x4 product R = M1 * M2 (matrixMult4Real, expmCuda.cu:1894-1917), each entry
// the first product then three fused multiply-adds; R may alias.
__device__ __forceinline__ void wmat4(const double *M1, const double *M2, double *R, int lane) {
    double t = 0.0;
    if (lane < 16) {
        int r = lane >> 2, c = lane & 3;
        t = M1[r * 4 + 0] * M2[0 * 4 + c];
        t = __fma_rn(M1[r * 4 + 1], M2[1 * 4 + c], t);
        t = __fma_rn(M1[r * 4 + 2], M2[2 * 4 + c], t);
        t = __fma_rn(M1[r * 4 + 3], M2[3 * 4 + c], t);
    }
    __syncwarp();
    if (lane < 16) R[lane] = t;
    __syncwarp();
}

// normalizeMat4RealSafe, expmCuda.cu:1955-1980, as the oracle states it: lengths
// through sqrtf, the old first column's length for the new one, products with
// the reciprocal lengths.  Lane i < 3 handles row i of the three columns.
__device__ __forceinline__ void wnormalize(double *T, int lane) {
    double len = 0.0;
    if (lane < 2) {
        int c = lane ? 2 : 0;
        double a = T[c], b = T[4 + c], e = T[8 + c];
        len = (double)sqrtf((float)__fma_rn(e, e, __fma_rn(b, b, a * a)));
    }
    double lenU = __shfl_sync(kFull, len, 0), lenW = __shfl_sync(kFull, len, 1);
    bool okU = lenU > 1e-8f, okW = lenW > 1e-8f;
    double il = 0.0;
    if (lane < 2 && (lane ? okW : okU)) il = 1.0 / len;
    double iu = __shfl_sync(kFull, il, 0), iw = __shfl_sync(kFull, il, 1);
    int i = lane < 3 ? lane : 0;
    double wi = okW ? T[4 * i + 2] * iw : (i == 2 ? 1.0 : 0.0);
    double vi = T[4 * i + 1];
    // crossproductReal (expmCuda.cu:1934-1938): component i uses rows ia, ib
    int ia = (i == 0) ? 1 : 0, ib = (i == 2) ? 1 : 2;
    double w_a = __shfl_sync(kFull, wi, ia), w_b = __shfl_sync(kFull, wi, ib);
    double v_a = __shfl_sync(kFull, vi, ia), v_b = __shfl_sync(kFull, vi, ib);
    // component 1 is v0 w2 - v2 w0 negated: written as -v0 w2 + v2 w0 so that
    // no fused result is negated (a negated zero sum would flip its sign)
    double ui = (i == 1) ? __fma_rn(-v_a, w_b, v_b * w_a) : __fma_rn(v_a, w_b, -(v_b * w_a));
    ui = okU ? ui * iu : (i == 0 ? 1.0 : 0.0);
    double u_a = __shfl_sync(kFull, ui, ia), u_b = __shfl_sync(kFull, ui, ib);
    double vn = (i == 1) ? __fma_rn(-w_a, u_b, w_b * u_a) : __fma_rn(w_a, u_b, -(w_b * u_a));
    __syncwarp();
    if (lane < 3) {
        T[4 * i] = ui;
        T[4 * i + 1] = vn;
        T[4 * i + 2] = wi;
    }
    __syncwarp();
}

// EXPOKIT's number of squarings, int(log2 ||A||_inf) + 2 truncated toward zero
// (at least 0), from the bits of the norm (the oracle evaluates it with frexp).
__device__ __forceinline__ int expm_squarings_bits(long long hb) {
    if (hb <= 0) return 0;
    int Eb = (int)(hb >> 52);
    if (Eb == 0) return 0;   // subnormal: far below 1
    if (Eb == 0x7ff) return 1;  // infinite norm (frexp leaves the exponent 0)
    bool frac0 = (hb & ((1LL << 52) - 1)) == 0;
    int tl = (Eb >= 1023) ? Eb - 1023 : (frac0 ? Eb - 1023 : Eb - 1022);
    int ns = tl + 2;
    return ns < 0 ? 0 : ns;
}

// exp(A) of a twist by the diagonal (6,6) Pade approximant with scaling and
// squaring (the method of EXPOKIT zgpadm used at expmCuda.cu:1642), real FP64.
// Result in S.E.
static __device__ void wexpm_twist(SolveScratch &S, const double *A, int lane) {
    long long sb = 0;
    if (lane < 4) {
        double s = fabs(A[lane * 4 + 0]);
        s = s + fabs(A[lane * 4 + 1]);
        s = s + fabs(A[lane * 4 + 2]);
        s = s + fabs(A[lane * 4 + 3]);
        sb = __double_as_longlong(s);
    }
    long long hb = 0;
#pragma unroll
    for (int r = 0; r < 4; r++) {
        long long v = __shfl_sync(kFull, sb, r);
        if (v <= kInfBits && v > hb) hb = v;  // NaN row sums never win, as in the oracle
    }
    int ns = expm_squarings_bits(hb);
    double scale = __longlong_as_double((long long)(1023 - ns) << 52);
    double *X = S.M[0], *X2 = S.M[1], *X4 = S.M[2], *X6 = S.M[3], *U0 = S.M[4], *V = S.M[5];
    if (lane < 16) X[lane] = A[lane] * scale;
    __syncwarp();
    wmat4(X, X, X2, lane);
    wmat4(X2, X2, X4, lane);
    wmat4(X4, X2, X6, lane);
    {
        // lanes 0-15: U0 = ((c1 I + c3 X2) + c5 X4) + 0 X6; lanes 16-31: V with c0, c2, c4, c6
        int e = lane & 15;
        bool isV = lane >= 16;
        double ca = isV ? kPade[0] : kPade[1], cb = isV ? kPade[2] : kPade[3];
        double cc = isV ? kPade[4] : kPade[5], cd = isV ? kPade[6] : 0.0;
        double I = (e % 5 == 0) ? 1.0 : 0.0;
        double o = __fma_rn(cd, X6[e], __fma_rn(cc, X4[e], __fma_rn(cb, X2[e], ca * I)));
        (isV ? V : U0)[e] = o;
    }
    __syncwarp();
    double *U = S.M[1];  // X2 no longer needed
    wmat4(X, U0, U, lane);
    double *Nm = S.M[2], *Dm = S.M[3];
    {
        int e = lane & 15;
        if (lane < 16) Nm[e] = V[e] + U[e];
        else Dm[e] = V[e] - U[e];
    }
    __syncwarp();
    // elimination over rows 0..2 (the last rows of D and N are exactly e4)
    int row = lane >> 3, col = lane & 7;  // col 0..3 -> D, 4..7 -> N
    for (int k = 0; k < 3; k++) {
        int p = k;
        long long best = abs_bits(Dm[k * 4 + k]);
        bool best_nan = best > kInfBits;
        for (int i = k + 1; i < 3; i++) {
            long long v = abs_bits(Dm[i * 4 + k]);
            if (!best_nan && v <= kInfBits && v > best) {
                best = v;
                p = i;
            }
        }
        if (best == 0) {  // singular: exp replaced by the identity, as the oracle does
            if (lane < 16) S.E[lane] = (lane % 5 == 0) ? 1.0 : 0.0;
            __syncwarp();
            return;
        }
        if (p != k) {
            double t = 0.0;
            int src = (row == k) ? p : k;
            bool sw = (row == k || row == p);
            if (sw) t = (col < 4) ? Dm[src * 4 + col] : Nm[src * 4 + col - 4];
            __syncwarp();
            if (sw) {
                if (col < 4) Dm[row * 4 + col] = t;
                else Nm[row * 4 + col - 4] = t;
            }
            __syncwarp();
        }
        double inv = 1.0 / Dm[k * 4 + k];
        double nv = 0.0;
        bool act = (row > k && row < 3) && (col >= 4 || col >= k + 1);
        if (act) {
            double f = Dm[row * 4 + k] * inv;
            if (col < 4) nv = __fma_rn(-f, Dm[k * 4 + col], Dm[row * 4 + col]);
            else nv = __fma_rn(-f, Nm[k * 4 + col - 4], Nm[row * 4 + col - 4]);
        }
        __syncwarp();
        if (act) {
            if (col < 4) Dm[row * 4 + col] = nv;
            else Nm[row * 4 + col - 4] = nv;
        }
        if (lane == 0) S.lu_inv[k] = inv;
        __syncwarp();
    }
    // column-oriented back substitution from row 3 up; lanes (row, c) of N
    int c = col - 4;
    for (int k = 3; k >= 1; k--) {
        double nv = 0.0;
        bool act = (col >= 4) && (row < k);
        if (act) nv = __fma_rn(-Dm[row * 4 + k], Nm[k * 4 + c], Nm[row * 4 + c]);
        __syncwarp();
        if (act) Nm[row * 4 + c] = nv;
        __syncwarp();
        if (col >= 4 && row == k - 1) Nm[row * 4 + c] = Nm[row * 4 + c] * S.lu_inv[k - 1];
        __syncwarp();
    }
    for (int k = 0; k < ns; k++) wmat4(Nm, Nm, Nm, lane);
    if (lane < 16) S.E[lane] = Nm[lane];
    __syncwarp();
}

// Entry (r, k) of a twist's 4x4 matrix as an index into SolveScratch::tw
// (x0..x5, -x0..-x5, 0), four bits each.
constexpr unsigned long long kTwistIndex = 0xccccull << 48 | 0x5c07ull << 32 | 0x46c2ull << 16 | 0x318cull;
__device__ __forceinline__ int twist_index(int r, int k) { return (int)(kTwistIndex >> (4 * (4 * r + k))) & 15; }

// 1 / len for a float len within 2^-19 of 1, rounded to nearest: with
// len = 1 + d 2^-24 the value 1 - d 2^-24 + d^2 2^-48 has at most 48 fraction
// bits, so it is a double, and it differs from 1 / len by less than 2^-56,
// below half a unit in the last place.  Integer operations only.
__device__ __forceinline__ double inverse_near_one(float len) {
    long long d = (int)((len - 1.0f) * 16777216.0f);  // exact
    long long n = (1LL << 48) - (d << 24) + d * d;     // the inverse in units of 2^-48
    long long above = (1023LL << 52) + ((n - (1LL << 48)) << 4), below = (1022LL << 52) + ((n - (1LL << 47)) << 5);
    return __longlong_as_double(n >= (1LL << 48) ? above : below);
}

// wnormalize of a matrix whose entry (r, c) lane r rs + off + c holds in w, for
// first and third columns of length 1 to 2^-19 (in FP32); lanes i < 3 return
// row i of the three columns.  The same operations as wnormalize: a length of
// exactly 1 needs no division and no products.  `extra` is multiplied with
// `scale` on lanes 3..5 beside the first product of the cross products (one
// instruction for both).  Returns false, and nothing else, for other lengths.
__device__ __forceinline__ bool wnormalize_near_one(double w, int rs, int off, int lane, double extra, double scale,
                                                    double &u, double &v, double &wz, double &scaled) {
    int c = lane & 3, i = lane < 3 ? lane : 0;
    double a = __shfl_sync(kFull, w, off + c), b = __shfl_sync(kFull, w, rs + off + c);
    double e = __shfl_sync(kFull, w, 2 * rs + off + c);
    float sf = (float)__fma_rn(e, e, __fma_rn(b, b, a * a));
    int ia = (i == 0) ? 1 : 0, ib = (i == 2) ? 1 : 2;
    double va = __shfl_sync(kFull, w, ia * rs + off + 1), vb = __shfl_sync(kFull, w, ib * rs + off + 1);
    double wi = __shfl_sync(kFull, w, i * rs + off + 2);
    float su = __shfl_sync(kFull, sf, 0), sw = __shfl_sync(kFull, sf, 2);
    double iu = 1.0;
    bool unit = su == 1.0f && sw == 1.0f;
    if (!unit) {
        float lu = sqrtf(su), lw = sqrtf(sw);
        if (!(fabsf(lu - 1.0f) <= 1.9073486e-6f && fabsf(lw - 1.0f) <= 1.9073486e-6f)) return false;
        iu = inverse_near_one(lu);
        wi = wi * inverse_near_one(lw);
    }
    double wa = __shfl_sync(kFull, wi, ia), wb = __shfl_sync(kFull, wi, ib);
    // component 1 of a cross product is formed with both signs turned, as in wnormalize
    double p = (lane < 3 ? vb : extra) * (lane < 3 ? wa : scale);
    scaled = p;
    double ui = __fma_rn(i == 1 ? -va : va, wb, i == 1 ? p : -p);
    if (!unit) ui = ui * iu;
    double ua = __shfl_sync(kFull, ui, ia), ub = __shfl_sync(kFull, ui, ib);
    p = wb * ua;
    v = __fma_rn(i == 1 ? -wa : wa, ub, i == 1 ? p : -p);
    u = ui;
    wz = wi;
    return true;
}

// wexpm_update for a small twist, every |x_k| in [2^-100, 2^-4): the same
// operations on the same values with what is known of them left out.  Such a
// twist needs no squarings (its norm is below 1/4), and no pivoting (the
// denominator's diagonal is above 0.99, its other entries below 0.04); the
// products with the exact zeros of X, of the last rows of its powers and of
// the last row of N change no value (every entry is far from underflow, a
// cancellation gives +0 with or without them, and the last row of the result
// is (+0, +0, +0, 1)).  Lane (row, half, c): the entry (row, c), half 0 of the
// denominator and half 1 of the numerator.  What bounds it is the FP64 pipe:
// 64 cycles an instruction whether or not it depends on the one before, so
// the products that wait for no exchange are issued while one is under way.
// S.T holds the pose in FP64.
static __device__ void wexpm_small(SolveScratch &S, const double *x, float *TF, double scaleOut, int lane) {
    int row = lane >> 3, half = (lane >> 2) & 1, c = lane & 3, e = row * 4 + c;
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < 6; k++) {
            S.tw[k] = x[k];
            S.tw[6 + k] = -x[k];
        }
        S.tw[12] = 0.0;
    }
    __syncwarp();
    // the two columns of row `row` of X other than the diagonal and the translation
    int k1 = row == 0 ? 1 : 0, k2 = row == 2 ? 1 : 2;
    double a1 = S.tw[twist_index(row, k1)], a2 = S.tw[twist_index(row, k2)], av = S.tw[twist_index(row, 3)];
    double b1 = S.tw[twist_index(k1, c)], b2 = S.tw[twist_index(k2, c)];
    double *X2 = S.M[0], *X4 = S.M[1], *U0 = S.M[2], *V = S.M[3];
    // even coefficients for the numerator's V (half 1), odd ones for U0 (half 0)
    double ca = c == row ? (half ? kPade[0] : kPade[1]) : 0.0, cb = half ? kPade[2] : kPade[3];
    double cc = half ? kPade[4] : kPade[5], cd = half ? kPade[6] : 0.0;
    double x2 = __fma_rn(a2, b2, a1 * b1);
    if (half == 0) X2[e] = x2;
    double o = __fma_rn(cb, x2, ca);
    __syncwarp();
    double r0 = X2[row * 4], r1 = X2[row * 4 + 1], r2 = X2[row * 4 + 2];
    double q0 = X2[c], q1 = X2[4 + c], q2 = X2[8 + c];
    double x4 = __fma_rn(r2, q2, __fma_rn(r1, q1, r0 * q0));
    if (half == 0) X4[e] = x4;
    o = __fma_rn(cc, x4, o);
    __syncwarp();
    r0 = X4[row * 4];
    r1 = X4[row * 4 + 1];
    r2 = X4[row * 4 + 2];
    double x6 = __fma_rn(r2, q2, __fma_rn(r1, q1, r0 * q0));
    o = __fma_rn(cd, x6, o);
    (half ? V : U0)[e] = o;
    __syncwarp();
    double un = __fma_rn(av, c == 3 ? kPade[1] : 0.0, __fma_rn(a2, U0[k2 * 4 + c], a1 * U0[k1 * 4 + c]));
    double w = V[e] + (half ? un : -un);
    // elimination of the denominator's rows 0..2 (column col of [D | N])
    int col = lane & 7;
    double f0 = __shfl_sync(kFull, w, row * 8), p0 = __shfl_sync(kFull, w, col);
    double i0 = 1.0 / __shfl_sync(kFull, w, 0);
    {
        double n = __fma_rn(-(f0 * i0), p0, w);
        if (row > 0 && row < 3 && col > 0) w = n;
    }
    double f1 = __shfl_sync(kFull, w, row * 8 + 1), p1 = __shfl_sync(kFull, w, 8 + col);
    double i1 = 1.0 / __shfl_sync(kFull, w, 9);
    {
        double n = __fma_rn(-(f1 * i1), p1, w);
        if (row == 2 && col > 1) w = n;
    }
    double d01 = __shfl_sync(kFull, w, 1), d2 = __shfl_sync(kFull, w, row * 8 + 2);
    double d3 = __shfl_sync(kFull, w, row * 8 + 3), n3 = __shfl_sync(kFull, w, 24 + col);
    double i2 = 1.0 / __shfl_sync(kFull, w, 18);
    // substitution from row 3 up, on the numerator's lanes
    bool num = half == 1;
    {
        double n = __fma_rn(-d3, n3, w);
        if (num && row < 3) w = n;
        n = w * i2;
        if (num && row == 2) w = n;
    }
    {
        double n = __fma_rn(-d2, __shfl_sync(kFull, w, 16 + col), w);
        if (num && row < 2) w = n;
        n = w * i1;
        if (num && row == 1) w = n;
    }
    {
        double n = __fma_rn(-d01, __shfl_sync(kFull, w, 8 + col), w);
        n = n * i0;
        if (num && row == 0) w = n;
    }
    // orthonormal columns, the translation scaled
    double t3 = __shfl_sync(kFull, w, (lane >= 3 && lane < 6 ? lane - 3 : 0) * 8 + 7), u, v, wz, sc;
    if (wnormalize_near_one(w, 8, 4, lane, t3, scaleOut, u, v, wz, sc)) {
        if (lane < 3) {
            S.Tinc[4 * lane] = u;
            S.Tinc[4 * lane + 1] = v;
            S.Tinc[4 * lane + 2] = wz;
        } else if (lane < 6) {
            S.Tinc[4 * (lane - 3) + 3] = sc;
        }
        __syncwarp();
    } else {
        if (num) S.Tinc[e] = row < 3 ? w : (c == 3 ? 1.0 : 0.0);
        __syncwarp();
        wnormalize(S.Tinc, lane);
        if (lane < 3) S.Tinc[4 * lane + 3] *= scaleOut;
        __syncwarp();
    }
    int tr = (lane >> 2) & 3;
    double t = S.T[tr * 4] * S.Tinc[c];
    t = __fma_rn(S.T[tr * 4 + 1], S.Tinc[4 + c], t);
    t = __fma_rn(S.T[tr * 4 + 2], S.Tinc[8 + c], t);
    t = __fma_rn(S.T[tr * 4 + 3], c == 3 ? 1.0 : 0.0, t);
    __syncwarp();
    if (lane < 16) S.T[lane] = t;
    if (wnormalize_near_one(t, 4, 0, lane, 0.0, 0.0, u, v, wz, sc)) {
        __syncwarp();
        if (lane < 3) {
            S.T[4 * lane] = u;
            S.T[4 * lane + 1] = v;
            S.T[4 * lane + 2] = wz;
        }
        __syncwarp();
    } else {
        __syncwarp();
        wnormalize(S.T, lane);
    }
    if (lane < 16) TF[lane] = (float)S.T[lane];
    __syncwarp();
}

// generateA + expmKernel (warp.cu:910-915, expmCuda.cu:1989-2048): T <- T * exp(A(x)),
// translation scaled by scaleOut, stored as float.  x is the same on every
// lane; TF is shared memory; S.T holds it in FP64.
static __device__ void wexpm_update(SolveScratch &S, const double *x, float *TF, double scaleOut, int lane) {
    // the largest |entry| is nonzero iff some x_k is nonzero and not NaN
    bool nonzero = false, small = true;
#pragma unroll
    for (int k = 0; k < 6; k++) {
        long long v = abs_bits(x[k]);
        nonzero |= (v != 0 && v <= kInfBits);
        small &= v >= (1023LL - 100) << 52 && v < (1023LL - 4) << 52;
    }
    // a Gauss-Newton step is small unless the start pose is far off (below
    // 1/16 rad and, with the reference's 1e-3 scale, 62 mm); then the chain of
    // FP64 instructions is about half as long as the general one
    if (small) {
        wexpm_small(S, x, TF, scaleOut, lane);
        return;
    }
    // the twist matrix lives in S.Tinc until exp(A) replaces it
    if (lane == 0) {
        double *A = S.Tinc;
        A[0] = 0.0; A[1] = -x[2]; A[2] = x[1]; A[3] = x[3];
        A[4] = x[2]; A[5] = 0.0; A[6] = -x[0]; A[7] = x[4];
        A[8] = -x[1]; A[9] = x[0]; A[10] = 0.0; A[11] = x[5];
        A[12] = 0.0; A[13] = 0.0; A[14] = 0.0; A[15] = 0.0;
    }
    __syncwarp();
    if (nonzero) {
        wexpm_twist(S, S.Tinc, lane);
        if (lane < 16) S.Tinc[lane] = S.E[lane];
        __syncwarp();
        wnormalize(S.Tinc, lane);
        if (lane < 3) S.Tinc[4 * lane + 3] *= scaleOut;
    } else {
        if (lane < 16) S.Tinc[lane] = (lane % 5 == 0) ? 1.0 : 0.0;
    }
    __syncwarp();
    wmat4(S.T, S.Tinc, S.T, lane);
    wnormalize(S.T, lane);
    if (lane < 16) TF[lane] = (float)S.T[lane];
    __syncwarp();
}

// Index of term (a, b), a <= b, of a packed symmetric 6x6 matrix
__device__ __forceinline__ int packed_base(int a) { return a * 6 - (a * (a - 1)) / 2 - a; }

// FP64 square-root-free Cholesky A = L D L^T with reciprocal pivots and
// column-oriented substitutions (orc_solve_cholesky).  Lane q < 21 holds the
// packed term (a, b), a <= b, of A in v and lanes 21..26 the right-hand side;
// x is returned on every lane.  A column's update is one fused multiply-add
// for all entries behind it and the right-hand side: each entry meets the
// same products in the same order as in the column-by-column form, and a
// column costs one reciprocal, one product and one multiply-add.  Returns 0,
// or -1 when a pivot is not positive.
static __device__ int wcholesky(double v, double *x, int lane) {
    int a = 0, b = lane;  // the lane's term: entry (row b, column a); right-hand side: row b, column 6
#pragma unroll
    for (int k = 1; k < 6; k++)
        if (lane >= packed_base(k) + k) {
            a = k;
            b = lane - packed_base(k);
        }
    if (lane >= 21) {
        a = 6;
        b = lane < 27 ? lane - 21 : 0;
    }
    double invrow = 0.0;  // right-hand side lanes: the reciprocal pivot of the row
    double lk[6];
#pragma unroll
    for (int j = 0; j < 6; j++) {
        double dj = __shfl_sync(kFull, v, packed_base(j) + j);
        long long bits = __double_as_longlong(dj);
        if (!(bits > 0 && bits <= kInfBits)) return -1;  // dj > 0
        double vb = __shfl_sync(kFull, v, packed_base(j) + (b > j ? b : j));
        double va = __shfl_sync(kFull, v, a == 6 ? 21 + j : packed_base(j) + (a > j ? a : j));
        if (j == 5) {
#pragma unroll
            for (int k = 1; k < 6; k++) lk[k] = __shfl_sync(kFull, v, packed_base(b < k ? b : k) + k);
        }
        double inv = 1.0 / dj;
        if (a == 6 && b == j) invrow = inv;
        double l = vb * inv;
        double n = __fma_rn(-l, va, v);
        if (b > j && a > j) v = n;
        if (a == j && b > j) v = l;  // the column of L
    }
    double z = v * invrow;
#pragma unroll
    for (int k = 5; k >= 1; k--) {
        double n = __fma_rn(-lk[k], __shfl_sync(kFull, z, 21 + k), z);
        if (b < k) z = n;
    }
#pragma unroll
    for (int k = 0; k < 6; k++) x[k] = __shfl_sync(kFull, z, 21 + k);
    return 0;
}

// conjugateGradientKernel, warp.cu:926-975, of S.A and S.b: at most 6 steps,
// tolerance 1e-8.  Lane j + 6 m evaluates the product A[j][m] dir[m] (and every
// lane A[j][5] dir[5]); the sums are then taken in the reference's order by
// every lane.  The squared residual of one step's end is the next one's start.
// sqrt(rr) < 1e-8 is rr < the smallest double whose rounded root reaches 1e-8.
static __device__ void wcg(const SolveScratch &S, double *x, int lane) {
    constexpr long long kTolBits = 0x3e45798ee2308c3aLL;  // 1e-8
    constexpr long long kRootBits = 0x3c9cd2b297d889bcLL;
    int j = lane % 6, m = lane / 6;
    double a1 = S.A[j * 6 + m], a2 = S.A[j * 6 + 5];
    double r = S.b[j], dir = r, xj = 0.0;
    auto no_negative_zero = [](double v) {  // 0.0 + v
        return __double_as_longlong(v) == (long long)0x8000000000000000ULL ? 0.0 : v;
    };
    auto sum6 = [&](double p) {
        double s = no_negative_zero(__shfl_sync(kFull, p, 0));
#pragma unroll
        for (int k = 1; k < 6; k++) s += __shfl_sync(kFull, p, k);
        return s;
    };
    double rr = sum6(r * r);
    for (int step = 0; step < 6; step++) {
        double p1 = a1 * __shfl_sync(kFull, dir, m), p2 = a2 * __shfl_sync(kFull, dir, 5);
        double ad = no_negative_zero(__shfl_sync(kFull, p1, j));
#pragma unroll
        for (int k = 1; k < 5; k++) ad += __shfl_sync(kFull, p1, j + 6 * k);
        ad += p2;
        double add = sum6(ad * dir);
        long long dv = abs_bits(add);
        double len = 0.0;
        if (dv > kTolBits && dv <= kInfBits) len = rr / add;
        r -= len * ad;
        double rr2 = sum6(r * r);
        xj += len * dir;
        if (abs_bits(rr2) < kRootBits) break;
        double beta = rr2 / rr;
        dir = r + beta * dir;
        rr = rr2;
    }
#pragma unroll
    for (int k = 0; k < 6; k++) x[k] = __shfl_sync(kFull, xj, k);
}

// Solves the packed system v (wcholesky's layout) and applies the update to
// TF (S.T: the same in FP64).  Returns the solve status.
static __device__ int wsolve_packed(SolveScratch &S, int solver, double v, float *TF, double scaleOut, int lane) {
    int st = 0;
    double x[6];
    if (solver == 1) {
        int a = 0, b = lane;
#pragma unroll
        for (int k = 1; k < 6; k++)
            if (lane >= packed_base(k) + k) {
                a = k;
                b = lane - packed_base(k);
            }
        if (lane < 21) {
            S.A[a * 6 + b] = v;
            S.A[b * 6 + a] = v;
        } else if (lane < 27) {
            S.b[lane - 21] = v;
        }
        __syncwarp();
        wcg(S, x, lane);
    } else {
        st = wcholesky(v, x, lane);
        if (st != 0) {
#pragma unroll
            for (int k = 0; k < 6; k++) x[k] = 0.0;
        }
    }
    wexpm_update(S, x, TF, scaleOut, lane);
    return st;
}

// Solve S.A x = S.b (A symmetric for the Cholesky solver) and apply the update
// to TF.  Returns the solve status.
static __device__ int wsolve_update(SolveScratch &S, int solver, float *TF, double scaleOut, int lane) {
    if (lane < 16) S.T[lane] = (double)TF[lane];
    __syncwarp();
    if (solver == 1) {
        double x[6];
        wcg(S, x, lane);
        wexpm_update(S, x, TF, scaleOut, lane);
        return 0;
    }
    int a = 0, b = lane;
#pragma unroll
    for (int k = 1; k < 6; k++)
        if (lane >= packed_base(k) + k) {
            a = k;
            b = lane - packed_base(k);
        }
    double v = lane < 21 ? S.A[b * 6 + a] : (lane < 27 ? S.b[lane - 21] : 0.0);
    return wsolve_packed(S, 0, v, TF, scaleOut, lane);
}

}  // namespace rt
