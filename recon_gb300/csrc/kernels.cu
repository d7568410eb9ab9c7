// kernels.cu -- sm_103a kernels of the dense RGB-D tracking hot path.
//
// Compiled with -fmad=false: every FP32/FP64 expression is rounded operation by
// operation in the reference's source order, so the results reproduce the
// reference semantics (and the CPU oracle) bit for bit.  One launch serves all
// tracker instances of a batch (blockIdx.y = instance).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstddef>
#include <mutex>

#include "scene.h"
#include "exact_arith.cuh"
#include "fx.cuh"
#include "pair_math.cuh"
#include "solve.cuh"
#include "track_kernels.cuh"
#include "track_math.cuh"

namespace rt {

#define INST_DESC const InstDesc &d = D[blockIdx.y]

// Copies an instance descriptor (pointers, sizes, calibration) into shared
// memory with one parallel load instead of a chain of dependent global loads.
__device__ __forceinline__ void load_desc(InstDesc &sd, const InstDesc *src_desc) {
    const int *src = reinterpret_cast<const int *>(src_desc);
    int *dst = reinterpret_cast<int *>(&sd);
    for (int k = threadIdx.x; k < (int)(sizeof(InstDesc) / sizeof(int)); k += blockDim.x) dst[k] = __ldg(src + k);
}

// ------------------------------------------------------------------
// input conversion and pyramids
// ------------------------------------------------------------------

// Back-projection with the IR camera, (x - cx) z / fx and (y - cy) z / fy: all
// pixels divide by the same focal lengths, so by their reciprocals and the exact
// division of pair_math.cuh.  (A pixel on the principal point's column or row, whose
// quotient is -0, takes the division.)
struct PixelRays {
    float fx, fy, cx, cy, rfx, rfy;
    bool plain;
    __device__ __forceinline__ explicit PixelRays(const float *KL) : fx(KL[0]), fy(KL[4]), cx(KL[2]), cy(KL[5]) {
        plain = div_in_range(fx, fy, fx);
        rfx = rcp_rn(fx);
        rfy = rcp_rn(fy);
    }
    __device__ __forceinline__ void point(int xi, int yi, float z, float &x, float &y) const {
        float ax = ((float)xi - cx) * z, ay = ((float)yi - cy) * z;
        x = div_rn(ax, -fx, rfx);
        y = div_rn(ay, -fy, rfy);
        if (!(plain && div_in_range(ax, ay, ax))) {
            x = ieee_div(ax, fx);
            y = ieee_div(ay, fy);
        }
    }
};

// three sums over ns = 1 .. 4 values into their means
__device__ __forceinline__ void mean3(float ns, float &a, float &b, float &c) {
    float y = rcp_rn(ns), qa = div_rn(a, -ns, y), qb = div_rn(b, -ns, y), qc = div_rn(c, -ns, y);
    if (!(div_in_range(a) && div_in_range(b) && div_in_range(c))) {
        qa = ieee_div(a, ns);
        qb = ieee_div(b, ns);
        qc = ieee_div(c, ns);
    }
    a = qa;
    b = qb;
    c = qc;
}

// The reference frame's level 0: uint8 gray -> [0,1], uint16 mm -> z = -mm
// (rgb2gray.cu:64-76 for the u8/u16 form, or the float4 RGBA+depth frame with
// its y-flip, rgbTex2GrayHdrZKernel); k_normals forms its points.  The current
// frame uses k_prep_current_pyramid.
__device__ __forceinline__ void convert_pixel(const InstDesc &d, const uint8_t *gp, const uint16_t *dp, const float *fp,
                                              int i, int xi, int yi, float &g, float &z) {
    if (fp) {
        // rgbTex2GrayHdrZKernel: texture read at (x, H-1-y)
        float4 p = __ldg((const float4 *)fp + xi + (d.H - 1 - yi) * d.W);
        g = 0.3f * p.x + 0.59f * p.y + 0.11f * p.z;
        float minDist = d.calib[RC_MIND], maxDist = d.calib[RC_MAXD];
        z = -(p.w * (maxDist - minDist) + minDist);
    } else {
        g = gray_unit(__ldg(gp + i));
        uint16_t dm = __ldg(dp + i);
        z = dm ? -(float)dm : 0.0f;
    }
}

__global__ void k_convert_level0(const InstDesc *D, const uint8_t *const *in_gray, const uint16_t *const *in_depth,
                                 const float *const *in_rgbd, int per_cta) {
    INST_DESC;
    const uint8_t *gp = in_gray[blockIdx.y];
    const uint16_t *dp = in_depth[blockIdx.y];
    const float *fp = in_rgbd[blockIdx.y];
    if (!fp && (!gp || !dp)) return;  // instance not updated by this call
    int n = d.W * d.H;
#pragma unroll 4
    for (int m = 0; m < per_cta; m += 256) {
        int i = blockIdx.x * per_cta + m + threadIdx.x;
        if (i >= n) return;
        float g, z;
        convert_pixel(d, gp, dp, fp, i, i % d.W, i / d.W, g, z);
        d.ref_gray[0][i] = g;
        d.ref_z[i] = z;
        d.ref_col[i] = -1.0f;  // a new keyframe has no fused colour
    }
}

// The current frame's whole pyramid in one pass: the level-0 conversion
// (convert_pixel, and genPointsCloud6Kernel, d2z.cu:436-469, for the cloud)
// and the 2x2 reductions of fastDownSampleHdrKernel and downSampleCloud6Kernel
// for the coarser levels (the expressions of k_downsample, in its order), so
// every value is identical to the separate kernels'.  A CTA of 256 threads
// takes a 32x32 tile of level 0: each thread converts one 2x2 block and reduces it
// to its level-1 pixel in registers; levels 2 and 3 come from the level-1 tile in
// shared memory.  Level 0 is never read back.  54 us for 30 640x480 frames, of which
// the bytes take 24; 68 with IEEE divisions and one pixel per access.
constexpr int kPyrTile = 32;

__device__ __forceinline__ void cloud_point(const PixelRays &rays, int xi, int yi, float z, float4 &o) {
    o = make_float4(0.f, 0.f, 0.f, 0.f);
    if (z < 0) {
        rays.point(xi, yi, z, o.x, o.y);
        o.z = z;
        o.w = 1.0f;
    }
}

// downSampleCloud6Kernel's average of the valid points among four (d2z.cu:557-588)
__device__ __forceinline__ float4 down_points(const float4 &a, const float4 &b, const float4 &c, const float4 &e) {
    float p0 = 0.0f, p1 = 0.0f, p2 = 0.0f, ns = 0.0f;
    const float4 *q[4] = {&a, &b, &c, &e};
#pragma unroll
    for (int k = 0; k < 4; k++) {
        if (q[k]->w != 0.0f) {
            ns++;
            p0 += q[k]->x;
            p1 += q[k]->y;
            p2 += q[k]->z;
        }
    }
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    if (ns > 0.0f) {
        mean3(ns, p0, p1, p2);
        o = make_float4(p0, p1, p2, 1.0f);
    }
    return o;
}

// In a sequence the kernel also does the per-frame bookkeeping in CTA 0 of
// each instance (saving two launches a frame): with `store_prev` it stores the
// previous frame's tracked pose (k_store_pose), with `begin` it resets the
// frame's statistics and sums (k_begin_track without an initial pose).
__global__ void __launch_bounds__(256) k_prep_current_pyramid(const InstDesc *D, const uint8_t *const *in_gray,
                                                              const uint16_t *const *in_depth,
                                                              const float *const *in_rgbd, int tiles_x,
                                                              float *store_prev, int begin) {
    __shared__ InstDesc sd;
    __shared__ float sg[2][256];   // gray of levels 1 (16x16) and 2 (8x8)
    __shared__ float4 sp[2][256];  // points of levels 1 and 2
    load_desc(sd, D + blockIdx.y);
    const uint8_t *gp = in_gray[blockIdx.y];
    const uint16_t *dp = in_depth[blockIdx.y];
    const float *fp = in_rgbd[blockIdx.y];
    __syncthreads();
    const InstDesc &d = sd;
    if (blockIdx.x == 0) {
        int t = threadIdx.x;
        if (store_prev && t < 16) store_prev[16 * blockIdx.y + t] = d.T[t];
        if (begin) {
            if (t < ST_COUNT) d.stats[t] = 0;
            if (t == 0) {
                *d.counter = 0u;
                if (d.trace_count) *d.trace_count = 0;
            }
            for (int k = t; k < 2 * 27 * kFxLimbs; k += blockDim.x) d.fx[k] = 0ull;
            if (t < 2) d.fx_bad[t] = 0;
        }
    }
    if (!fp && (!gp || !dp)) return;  // instance not updated by this call
    int W = d.W, H = d.H;
    int tx = blockIdx.x % tiles_x, ty = blockIdx.x / tiles_x;
    if (tx * kPyrTile >= W || ty * kPyrTile >= H) return;
    int t = threadIdx.x;
    int bx = t % 16, by = t / 16;
    int x0 = tx * kPyrTile + 2 * bx, y0 = ty * kPyrTile + 2 * by;
    // level 0: the 2x2 block (x0, y0) .. (x0 + 1, y0 + 1), in k_downsample's order
    float g[4];
    float4 pt[4];
    bool in0 = x0 < W && y0 < H;
    const PixelRays rays(d.calib + RC_KL);
    // pixels in pairs where the width is even and the inputs are aligned to it
    if (in0 && !fp && !(W & 1) && !(reinterpret_cast<uintptr_t>(gp) & 1) && !(reinterpret_cast<uintptr_t>(dp) & 3)) {
#pragma unroll
        for (int r = 0; r < 2; r++) {
            g[2 * r] = g[2 * r + 1] = 0.0f;
            pt[2 * r] = pt[2 * r + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (y0 + r >= H) continue;
            int i = x0 + (y0 + r) * W;
            uchar2 gg = __ldg(reinterpret_cast<const uchar2 *>(gp + i));
            ushort2 dd = __ldg(reinterpret_cast<const ushort2 *>(dp + i));
            float2 gf = make_float2(gray_unit(gg.x), gray_unit(gg.y));
            float2 z = make_float2(dd.x ? -(float)dd.x : 0.0f, dd.y ? -(float)dd.y : 0.0f);
            *reinterpret_cast<float2 *>(d.cur_gray[0] + i) = gf;
            *reinterpret_cast<float2 *>(d.cur_z + i) = z;
            if (d.cur_grayh[0]) *reinterpret_cast<__half2 *>(d.cur_grayh[0] + i) = __floats2half2_rn(gf.x, gf.y);
            g[2 * r] = gf.x;
            g[2 * r + 1] = gf.y;
            cloud_point(rays, x0, y0 + r, z.x, pt[2 * r]);
            cloud_point(rays, x0 + 1, y0 + r, z.y, pt[2 * r + 1]);
        }
    } else if (in0) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            int xi = x0 + (k & 1), yi = y0 + (k >> 1);
            g[k] = 0.0f;
            pt[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (xi >= W || yi >= H) continue;
            int i = xi + yi * W;
            float z;
            convert_pixel(d, gp, dp, fp, i, xi, yi, g[k], z);
            cloud_point(rays, xi, yi, z, pt[k]);
            d.cur_gray[0][i] = g[k];
            if (d.cur_grayh[0]) d.cur_grayh[0][i] = __float2half_rn(g[k]);  // mixed precision
            d.cur_z[i] = z;
        }
    }
    if (d.L < 2) return;
    // level 1 in registers (its pixel exists iff the whole block does)
    int w1 = W >> 1, h1 = H >> 1;
    int x1 = x0 >> 1, y1 = y0 >> 1;
    if (in0 && x1 < w1 && y1 < h1) {
        float gl = (g[0] + g[1] + g[2] + g[3]) / 4.0f;
        float4 o = down_points(pt[0], pt[1], pt[2], pt[3]);
        int i = x1 + y1 * w1;
        d.cur_gray[1][i] = gl;
        if (d.cur_grayh[1]) d.cur_grayh[1][i] = __float2half_rn(gl);
        d.cur_pts[1][i] = o;
        sg[0][t] = gl;
        sp[0][t] = o;
    }
    // levels 2 and 3 from the 16x16 level-1 tile (slot 0), level 2 in slot 1
    int side = 16;
    for (int l = 2; l < d.L; l++) {
        __syncthreads();
        int src = (l - 2) & 1;
        int hs = side;
        side >>= 1;
        int wl = W >> l, hl = H >> l;
        if (t < side * side) {
            int ox = t % side, oy = t / side;
            int gx = tx * (kPyrTile >> l) + ox, gy = ty * (kPyrTile >> l) + oy;
            if (gx < wl && gy < hl) {
                int c0 = 2 * ox + 2 * oy * hs;
                float gl = (sg[src][c0] + sg[src][c0 + 1] + sg[src][c0 + hs] + sg[src][c0 + hs + 1]) / 4.0f;
                float4 o = down_points(sp[src][c0], sp[src][c0 + 1], sp[src][c0 + hs], sp[src][c0 + hs + 1]);
                int i = gx + gy * wl;
                d.cur_gray[l][i] = gl;
                if (d.cur_grayh[l]) d.cur_grayh[l][i] = __float2half_rn(gl);
                d.cur_pts[l][i] = o;
                sg[1 - src][t] = gl;
                sp[1 - src][t] = o;
            }
        }
    }
}

// the ICP kernels' copy of reference pixel i: z NaN where the mask is 0
__device__ __forceinline__ void store_ref_planes(float *pl, int i, float x, float y, float z, float mask, float nx,
                                                 float ny, float nz) {
    float *o = pl + ref_plane(i, 0);
    o[0] = x;
    o[kChunk] = y;
    o[2 * kChunk] = mask != 0.0f ? z : __int_as_float(0x7fffffff);
    o[3 * kChunk] = nx;
    o[4 * kChunk] = ny;
    o[5 * kChunk] = nz;
}

// fastDownSampleHdrKernel (downSample2Cuda.cu:35-42) for the reference gray
// pyramid and downSampleCloud6Kernel (d2z.cu:557-588) for its point and normal
// pyramid.
__global__ void k_downsample(const InstDesc *D, int level, const int *active) {
    INST_DESC;
    if (!active[blockIdx.y]) return;
    if (level >= d.L) return;
    int wlo = d.W >> level, hlo = d.H >> level;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= wlo * hlo) return;
    int x = i % wlo, y = i / wlo;
    int w2 = 2 * wlo;
    int h0 = 2 * x + 2 * y * w2;
    const float *hi = d.ref_gray[level - 1];
    d.ref_gray[level][i] = (hi[h0] + hi[h0 + 1] + hi[h0 + w2] + hi[h0 + w2 + 1]) / 4.0f;

    const float4 *src = d.ref_pts[level - 1];
    int offs[4] = {h0, h0 + 1, h0 + w2, h0 + w2 + 1};
    float p0 = 0.0f, p1 = 0.0f, p2 = 0.0f, n0 = 0.0f, n1 = 0.0f, n2 = 0.0f;
    float ns = 0.0f;
    for (int k = 0; k < 4; k++) {
        float4 s = src[offs[k]];
        if (s.w != 0.0f) {
            ns++;
            p0 += s.x;
            p1 += s.y;
            p2 += s.z;
            float4 nn = d.ref_nrm[level - 1][offs[k]];
            n0 += nn.x;
            n1 += nn.y;
            n2 += nn.z;
        }
    }
    if (ns > 0.0f) {
        mean3(ns, p0, p1, p2);
        mean3(ns, n0, n1, n2);
        normalize3(n0, n1, n2);
        d.ref_nrm[level][i] = make_float4(n0, n1, n2, 0.0f);
        d.ref_pts[level][i] = make_float4(p0, p1, p2, 1.0f);
        store_ref_planes(d.ref_pl[level], i, p0, p1, p2, 1.0f, n0, n1, n2);
    } else {
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
        d.ref_pts[level][i] = o;
        d.ref_nrm[level][i] = o;
        store_ref_planes(d.ref_pl[level], i, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f);
    }
}

// 1 / v, rounded once
__device__ __forceinline__ float reciprocal(float v) {
    float a = fabsf(v);
    return a >= kDivLo && a <= kDivHi ? rcp_rn(v) : ieee_div(1.0f, v);
}

// Gray value the RGB camera sees at point (qx, qy, qz) of its rig's IR frame
// (TLR, distortPoint and the bilinear color1 tap of xyz2CloudKernel,
// d2z.cu:235-331, with the perspective division as one reciprocal and two
// products), from a float image or a uint8 image scaled by 1/255; -1 where
// the 2x2 taps leave the image.  Used by the keyframe fusion only.
template <typename TImg>
__device__ __forceinline__ float rgb_sample(const float *calib, float qx, float qy, float qz, const TImg *img, int W,
                                            int H) {
    float rx, ry, rz;
    mul4(calib + RC_TLR, qx, qy, qz, rx, ry, rz);
    float irz = reciprocal(rz);
    float pux = rx * irz, puy = ry * irz;
    float px, py;
    distort(pux, puy, calib + RC_KCR, calib + RC_KR, px, py);
    int xdi = ftoi(px), ydi = ftoi(py);
    if (!(xdi >= 0 && ydi >= 0 && xdi < W - 1 && ydi < H - 1)) return -1.0f;
    float fx = px - xdi, fy = py - ydi;
    return bilin(xdi, ydi, fx, fy, W, img);
}

// Keyframe depth and colour fusion (the oracle's orc_fuse_rgbd restates the
// same steps): every valid keyframe pixel is back-projected with KL
// (rgb2gray.cu:570-593), mapped into frame f by its tracked pose, looked up at
// the nearest IR pixel (the zWeight tap of warp.cu:306-327), mapped back with
// the inverse pose (as filterDepthIIRKernel does, warp.cu:398-467), gated on
// |dz| < gate and averaged with unit weights (the running mean of
// updateVoxelsKernel, VoxelGrid_cuda.cu:1005-1013).  The divisions are
// written as products with reciprocals (of fx, fy per instance, of the
// depth once per projection); the oracle states the same.  With gray images the
// vertex colour is fused under the same gate: the mean of the keyframe's own
// sample at the point and the accepted frames' samples at T_f p
// (KeyFrameModel::integrateDepthMaps warps the neighbours' RGB images into the
// keyframe, KeyFrameModel.cpp:537-583).  Writes the fused depth in place into
// ref_z and the colour into ref_col (-1 where no sample exists).
// depth / gray: nframes x n_inst frame pointers (gray may be null: depth only,
// colours kept); Tf: nframes x n_inst x 16 poses.
// 8 CTAs per SM (32 registers, a few bytes of spill): more warps to hide the
// per-frame gathers, 402 us per 30 x 5-frame launch (471 us with IEEE reciprocals and
// divisions by 255)
#ifndef RECON_FUSE_MIN_BLOCKS
#define RECON_FUSE_MIN_BLOCKS 8
#endif
__global__ void __launch_bounds__(256, RECON_FUSE_MIN_BLOCKS) k_fuse_depth(const InstDesc *D, int nframes, int n_inst, const uint16_t *const *depth,
                             const uint8_t *const *gray, const float *Tf, float gate, const int *active) {
    INST_DESC;
    if (!active[blockIdx.y]) return;
    __shared__ float sT[8][16], sTi[8][16];
    if (threadIdx.x < nframes && threadIdx.x < 8) {
        const float *M = Tf + ((size_t)threadIdx.x * n_inst + blockIdx.y) * 16;
        float *Mi = sTi[threadIdx.x];
        for (int k = 0; k < 16; k++) sT[threadIdx.x][k] = M[k];
        // invertRT4Cuda, kernelUtils.h:100-107
        Mi[0] = M[0]; Mi[1] = M[4]; Mi[2] = M[8];   Mi[3] = -(M[0] * M[3] + M[4] * M[7] + M[8] * M[11]);
        Mi[4] = M[1]; Mi[5] = M[5]; Mi[6] = M[9];   Mi[7] = -(M[1] * M[3] + M[5] * M[7] + M[9] * M[11]);
        Mi[8] = M[2]; Mi[9] = M[6]; Mi[10] = M[10]; Mi[11] = -(M[2] * M[3] + M[6] * M[7] + M[10] * M[11]);
        Mi[12] = 0;   Mi[13] = 0;   Mi[14] = 0;     Mi[15] = 1;
    }
    __syncthreads();
    int W = d.W, H = d.H;
    int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= W * H) return;
    float minDist = d.calib[RC_MIND], maxDist = d.calib[RC_MAXD];
    const float *KL = d.calib + RC_KL;
    float fx = KL[0], fy = KL[4], cx = KL[2], cy = KL[5];
    float ifx = 1.0f / fx, ify = 1.0f / fy;
    int xi = idx % W, yi = idx / W;
    float z = d.ref_z[idx];
    const bool colour = gray != nullptr;
    if (!(z < -minDist && z > -maxDist)) {
        if (colour) d.ref_col[idx] = -1.0f;
        return;
    }
    float px3 = ((float)xi - cx) * z * ifx, py3 = ((float)yi - cy) * z * ify, pz3 = z;
    float zsum = z, wsum = 1.0f;
    float csum = 0.0f, cw = 0.0f;
    if (colour) {
        float c0 = rgb_sample(d.calib, px3, py3, pz3, d.ref_gray[0], W, H);
        if (c0 >= 0.0f) {
            csum = c0;
            cw = 1.0f;
        }
    }
    for (int f = 0; f < nframes && f < 8; f++) {
        float qx, qy, qz;
        mul4(sT[f], px3, py3, pz3, qx, qy, qz);
        float iqz = reciprocal(qz);
        float q2x = qx * iqz, q2y = qy * iqz;
        float pxl = KL[0] * q2x + KL[1] * q2y + KL[2];
        float pyl = KL[3] * q2x + KL[4] * q2y + KL[5];
        int xd = ftoi(pxl + 0.5f), yd = ftoi(pyl + 0.5f);
        if (xd < 0 || yd < 0 || xd >= W || yd >= H) continue;
        uint16_t dm = depth[(size_t)f * n_inst + blockIdx.y][xd + yd * W];
        float zf = dm ? -(float)dm : 0.0f;
        if (!(zf < -minDist && zf > -maxDist)) continue;
        float mx = ((float)xd - cx) * zf * ifx, my = ((float)yd - cy) * zf * ify, mz = zf;
        float kx, ky, kz;
        mul4(sTi[f], mx, my, mz, kx, ky, kz);
        float dz = kz - z;
        if (fabsf(dz) < gate) {
            zsum += kz;
            wsum += 1.0f;
            if (colour) {
                float c = rgb_sample(d.calib, qx, qy, qz, gray[(size_t)f * n_inst + blockIdx.y], W, H);
                if (c >= 0.0f) {
                    csum += c;
                    cw += 1.0f;
                }
            }
        }
    }
    d.ref_z[idx] = zsum / wsum;
    if (colour) d.ref_col[idx] = cw > 0.0f ? csum / cw : -1.0f;
}

// genOrientedPoints6Kernel (d2z.cu:471-501): the filtered reference's level-0
// ICP points and normals from a ray-cast point image and its normals (float4
// maps of the keyframe's pixels, camera frame); replaces what k_normals wrote
// for the instances whose point pointer is set
__global__ void k_oriented_points(const InstDesc *D, const float *const *in_pts, const float *const *in_nrm) {
    INST_DESC;
    const float4 *pts = reinterpret_cast<const float4 *>(in_pts[blockIdx.y]);
    const float4 *nrm = reinterpret_cast<const float4 *>(in_nrm[blockIdx.y]);
    if (!pts || !nrm) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.W * d.H) return;
    const float4 v = pts[i], n = nrm[i];
    const float len = n.x * n.x + n.y * n.y + n.z * n.z;
    if (v.z < 0 && len > 1e-7f) {
        d.ref_pts[0][i] = make_float4(v.x, v.y, v.z, 1.0f);
        d.ref_nrm[0][i] = make_float4(n.x, n.y, n.z, 0.0f);
        store_ref_planes(d.ref_pl[0], i, v.x, v.y, v.z, 1.0f, n.x, n.y, n.z);
    } else {
        d.ref_pts[0][i] = make_float4(0.f, 0.f, 0.f, 0.f);
        d.ref_nrm[0][i] = make_float4(0.f, 0.f, 0.f, 0.f);
        store_ref_planes(d.ref_pl[0], i, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f);
    }
}

// The reference's level-0 ICP point of a keyframe pixel of depth z
// (convertZMapToXYZ6Kernel, rgb2gray.cu:595-624; the same formula as
// convertZMapToXYZKernel, 570-593): zero out of range.
__device__ __forceinline__ float4 ref_point(const InstDesc &d, const PixelRays &rays, int xi, int yi, float z) {
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    if (z < -d.calib[RC_MIND] && z > -d.calib[RC_MAXD]) {
        rays.point(xi, yi, z, o.x, o.y);
        o.z = z;
        o.w = 1.0f;
    }
    return o;
}

// The reference's level 0 from the keyframe depth: the points, and their normals
// and masks (computeNormalsCudaKernel, d2z.cu:503-537).  It is bound by the 56
// bytes that it writes per pixel; a pixel's four neighbours are formed from their
// depths again, which costs less than reading points that another kernel wrote
// (30 640x480 frames: 108 us here and 39 for the conversion; 105 and 80 where the
// conversion writes the points, and a launch of 52 us to form those of a fused depth).
__global__ void k_normals(const InstDesc *D, const int *active, int per_cta) {
    INST_DESC;
    if (!active[blockIdx.y]) return;
    int W = d.W, H = d.H;
    const PixelRays rays(d.calib + RC_KL);
    const float *z = d.ref_z;
    for (int m = 0; m < per_cta; m += 256) {
        int i = blockIdx.x * per_cta + m + threadIdx.x;
        if (i >= W * H) return;
        int xi = i % W, yi = i / W;
        float4 me = ref_point(d, rays, xi, yi, z[i]), nrm = make_float4(0.f, 0.f, 0.f, 0.f);
        float mask = 0.0f;
        if (!(xi < 1 || yi < 1 || xi > W - 2 || yi > H - 2)) {
            float4 x1 = ref_point(d, rays, xi - 1, yi, z[i - 1]), x2 = ref_point(d, rays, xi + 1, yi, z[i + 1]);
            float4 y1 = ref_point(d, rays, xi, yi - 1, z[i - W]), y2 = ref_point(d, rays, xi, yi + 1, z[i + W]);
            if (x1.z < 0 && x2.z < 0 && y1.z < 0 && y2.z < 0) {
                float ux = x2.x - x1.x, uy = x2.y - x1.y, uz = x2.z - x1.z;
                float vx = y2.x - y1.x, vy = y2.y - y1.y, vz = y2.z - y1.z;
                float nx = uy * vz - uz * vy;
                float ny = -(ux * vz - uz * vx);
                float nz = ux * vy - uy * vx;
                normalize3(nx, ny, nz);
                nrm = make_float4(nx, ny, nz, 0.0f);
                mask = me.w;
            }
        }
        d.ref_nrm[0][i] = nrm;
        d.ref_pts[0][i] = make_float4(me.x, me.y, me.z, mask);
        store_ref_planes(d.ref_pl[0], i, me.x, me.y, me.z, mask, nrm.x, nrm.y, nrm.z);
    }
}

// ------------------------------------------------------------------
// photometric reference: vertex records, gradient histogram, selection
// ------------------------------------------------------------------

// The vertex record of keyframe pixel i (xyz2CloudKernel, d2z.cu:235-331):
// v = x y z px py gx gy gmag gray, zero with z = -maxDist where the point is
// invalid or projects within 10 pixels of the border.  The keyframe kernels
// evaluate it twice with the same operations: for every pixel to find the
// gradient magnitude that selects the points, and again for the selected
// points only (so that the other eight planes are never stored).  The point
// is the back-projection of the keyframe depth ref_z, formed as k_normals forms
// the level-0 ICP points (zero out of
// range: xyz alone carries the validity), so a filtered reference's oriented
// points, which later replace those, do not enter it.
__device__ __forceinline__ void vertex_record(const InstDesc &d, int i, int W, int H, float *v) {
    for (int k = 0; k < kVtxPlanes; k++) v[k] = 0.0f;
    v[2] = -d.calib[RC_MAXD];
    float p3x = 0.0f, p3y = 0.0f, p3z = 0.0f;
    {
        float z = d.ref_z[i];
        float minDist = d.calib[RC_MIND], maxDist = d.calib[RC_MAXD];
        if (z < -minDist && z > -maxDist) {
            PixelRays(d.calib + RC_KL).point(i % W, i / W, z, p3x, p3y);
            p3z = z;
        }
    }
    if (p3z < 0) {
        const float *T = d.calib + RC_TLR;
        float rx, ry, rz;
        mul4(T, p3x, p3y, p3z, rx, ry, rz);
        float irz = rcp_rn(rz), pux = div_rn(rx, -rz, irz), puy = div_rn(ry, -rz, irz);
        if (!div_in_range(rx, ry, rz)) {
            pux = ieee_div(rx, rz);
            puy = ieee_div(ry, rz);
        }
        float px, py;
        distort(pux, puy, d.calib + RC_KCR, d.calib + RC_KR, px, py);
        if (in_bounds10(px, py, W, H)) {
            const float *img = d.ref_gray[0];
            int xdi = ftoi(px), ydi = ftoi(py);
            float fx = px - xdi, fy = py - ydi;
            float color1, colorN, colorE, colorW, colorS;
            if (ftoi(px + 1.0f) == xdi + 1 && ftoi(px - 1.0f) == xdi - 1 && ftoi(py + 1.0f) == ydi + 1 &&
                ftoi(py - 1.0f) == ydi - 1) {
                // the five interpolations share 12 taps and their weights
                float w0 = (1 - fx) * (1 - fy), w1 = fx * (1 - fy), w2 = (1 - fx) * fy, w3 = fx * fy;
                const float *q = img + xdi + ydi * W;
                float a1 = __ldg(q - W), a2 = __ldg(q - W + 1);
                float b0 = __ldg(q - 1), b1 = __ldg(q), b2 = __ldg(q + 1), b3 = __ldg(q + 2);
                float c0 = __ldg(q + W - 1), c1 = __ldg(q + W), c2 = __ldg(q + W + 1), c3 = __ldg(q + W + 2);
                float e1 = __ldg(q + 2 * W), e2 = __ldg(q + 2 * W + 1);
                color1 = w0 * b1 + w1 * b2 + w2 * c1 + w3 * c2;
                colorN = w0 * a1 + w1 * a2 + w2 * b1 + w3 * b2;
                colorE = w0 * b2 + w1 * b3 + w2 * c2 + w3 * c3;
                colorW = w0 * b0 + w1 * b1 + w2 * c0 + w3 * c1;
                colorS = w0 * c1 + w1 * c2 + w2 * e1 + w3 * e2;
            } else {  // a coordinate that one more rounding takes to the next pixel
                color1 = bilin(xdi, ydi, fx, fy, W, img);
                colorN = bilin(ftoi(px), ftoi(py - 1.0f), fx, fy, W, img);
                colorE = bilin(ftoi(px + 1.0f), ftoi(py), fx, fy, W, img);
                colorW = bilin(ftoi(px - 1.0f), ftoi(py), fx, fy, W, img);
                colorS = bilin(ftoi(px), ftoi(py + 1.0f), fx, fy, W, img);
            }
            float fused = d.ref_col[i];  // the keyframe fusion's vertex colour, if any
            if (fused >= 0.0f) color1 = fused;
            float gradX1 = (colorE - colorW) / 2.0f;
            float gradY1 = (colorS - colorN) / 2.0f;
            float gm = fabsf(gradY1) + fabsf(gradX1);
            v[0] = p3x; v[1] = p3y; v[2] = p3z;
            v[3] = px; v[4] = py;
            v[5] = gradX1; v[6] = gradY1;
            v[7] = gm < 1.0f ? gm : 1.0f;
            v[8] = color1;
        }
    }
}

// The gradient magnitude of every keyframe pixel (xyz2CloudKernel's gmag
// plane) and its 256-bin histogram (gpu_hist.cu:136, cuda_hist.cu:100-152)
// with privatised shared-memory integer atomics.  Bound by the gathers of its 12
// taps and by the bins that each CTA adds to the instance's: 256 mixed frames
// 272 us with four pixels a thread, 466 with one, 20 taps and IEEE divisions.
__global__ void k_xyz2cloud(const InstDesc *D, const int *active, int per_cta) {
    INST_DESC;
    if (!active[blockIdx.y]) return;
    __shared__ int sh[1024];
    int nb = d.select_bins;
    for (int k = threadIdx.x; k < nb; k += blockDim.x) sh[k] = 0;
    __syncthreads();
    int W = d.W, H = d.H, n = W * H;
    for (int i = blockIdx.x * per_cta + threadIdx.x; i < min(n, ((int)blockIdx.x + 1) * per_cta); i += blockDim.x) {
        float v[kVtxPlanes];
        vertex_record(d, i, W, H, v);
        d.gmag[i] = v[7];
        unsigned int bin = (unsigned int)(v[7] * (nb - 1) + 0.5f);
        if (bin < (unsigned)nb) atomicAdd(&sh[bin], 1);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < nb; k += blockDim.x)
        if (sh[k]) atomicAdd(&d.grad_hist[k], sh[k]);
}

// seekThreshold256Kernel2 (filterIndex256.cu:26-46) + per-segment counts of
// filterIndexKernel4 (filterIndex256.cu:110-133).  seg layout:
// [0,512) cnt, [512,1024) mcnt, [1024,1536) start, [1536,2048) mstart,
// [2048,2560) kept, [3072] thr, [3073] excess, [3074] written.
__global__ void k_seg_count(const InstDesc *D, const int *active) {
    INST_DESC;
    if (!active[blockIdx.y]) return;
    int nb = d.select_bins, P = d.P;
    __shared__ unsigned int s_thr;
    __shared__ int s_excess;
    __shared__ int s_hist[1024];
    // the histogram in shared memory in one parallel load; the threshold
    // search (from the top bin down) then reads shared memory only
    for (int k = threadIdx.x; k < nb; k += blockDim.x) s_hist[k] = __ldcg(d.grad_hist + k);
    __syncthreads();
    if (threadIdx.x < 32) {
        // from the top bin down, 32 bins at a time: the first at which the running
        // count passes P (bin 0 when none does)
        int above = 0, thr = 0, sel = 0, l = threadIdx.x;
        for (int top = nb - 1;; top -= 32) {
            int k = top - l, incl = k >= 0 ? s_hist[k] : 0;
            for (int o = 1; o < 32; o <<= 1) {
                int t = __shfl_up_sync(0xffffffffu, incl, o);
                if (l >= o) incl += t;
            }
            unsigned past = __ballot_sync(0xffffffffu, above + incl > P);
            if (past || top < 32) {
                int first = past ? __ffs(past) - 1 : 31;
                sel = above + __shfl_sync(0xffffffffu, incl, first);
                thr = past ? top - first : 0;
                break;
            }
            above += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (l == 0) {
            s_thr = (unsigned)thr;
            s_excess = sel - P;
            if (blockIdx.x == 0) {
                d.seg[3072] = thr;
                d.seg[3073] = sel - P;
            }
        }
    }
    __syncthreads();
    int n = d.W * d.H;
    int ppt = n / kSegments;
    int warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    int lane = threadIdx.x & 31;
    if (warp >= kSegments) return;
    const float *grad = d.gmag;
    unsigned int thr = s_thr;
    int cnt = 0, mcnt = 0;
#pragma unroll 4
    for (int base = warp * ppt; base < warp * ppt + ppt; base += 32) {
        int i = base + lane;
        bool in = i < warp * ppt + ppt;
        unsigned int q = in ? (unsigned int)(__ldg(grad + i) * (nb - 1) + 0.5f) : 0u;
        cnt += in && q > thr;
        mcnt += in && q == thr;
    }
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    mcnt = __reduce_add_sync(0xffffffffu, mcnt);
    if (lane == 0) {
        d.seg[warp] = cnt;
        d.seg[512 + warp] = mcnt;
    }
}

// Exclusive prefix sum of kSegments (512) values in shared memory by the
// CTA's 512 threads: warp scans by shuffles, then the warps' totals.
__device__ __forceinline__ int block_exclusive_scan512(int v, int *warp_tot) {
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) warp_tot[w] = incl;
    __syncthreads();
    if (w == 0) {
        int t = lane < kSegments / 32 ? warp_tot[lane] : 0;
        int ti = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int u = __shfl_up_sync(0xffffffffu, ti, o);
            if (lane >= o) ti += u;
        }
        if (lane < kSegments / 32) warp_tot[lane] = ti - t;  // exclusive warp offsets
    }
    __syncthreads();
    return warp_tot[w] + incl - v;
}

// segment start offsets and the reference's sequential trimming of surplus
// threshold-bin points (filterIndex256.cu:136-157), one CTA of kSegments
// threads per instance: the start offsets are an exclusive prefix sum of the
// counts; the trimming walks the segments in order only while a surplus is
// left (after that it changes nothing), then the threshold-bin offsets are
// an exclusive prefix sum of what was kept, after the last start.
__global__ void k_seg_scan(const InstDesc *D, const int *active) {
    INST_DESC;
    if (!active[blockIdx.y]) return;
    __shared__ int s_kept[kSegments];
    __shared__ int warp_tot[kSegments / 32];
    int t = threadIdx.x;
    int *cnt = d.seg, *mcnt = d.seg + 512, *start = d.seg + 1024, *mstart = d.seg + 1536, *kept = d.seg + 2048;
    int c = __ldcg(cnt + t);
    s_kept[t] = __ldcg(mcnt + t);
    int st = block_exclusive_scan512(c, warp_tot);  // synchronises: s_kept is complete
    start[t] = st;
    if (t == 0) {
        int tooMuch = __ldcg(d.seg + 3073);
        for (int i = 1; i < kSegments && tooMuch > 0; i++) {
            if (s_kept[i - 1] > 0) {
                s_kept[i - 1] -= tooMuch;
                if (s_kept[i - 1] < 0) {
                    tooMuch += s_kept[i - 1];
                    s_kept[i - 1] = 0;
                } else {
                    tooMuch = 0;
                }
            }
        }
    }
    __syncthreads();
    // the total of the counts (the last start plus the last count) begins the threshold-bin offsets
    __shared__ int s_base;
    if (t == kSegments - 1) s_base = st + c;
    int k = s_kept[t];
    int ms = block_exclusive_scan512(k, warp_tot);  // synchronises: s_base is visible
    mstart[t] = s_base + ms;
    kept[t] = k;
    if (t == kSegments - 1) d.seg[3074] = s_base + ms + k;
}

// filterIndexKernel4's scatter (filterIndex256.cu:159-168): one warp per segment
__global__ void k_seg_scatter(const InstDesc *D, const int *active) {
    INST_DESC;
    if (!active[blockIdx.y]) return;
    int nb = d.select_bins, P = d.P;
    int n = d.W * d.H;
    int ppt = n / kSegments;
    int warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    int lane = threadIdx.x & 31;
    if (warp >= kSegments) return;
    const float *grad = d.gmag;
    unsigned int thr = (unsigned int)d.seg[3072];
    int pos_a = d.seg[1024 + warp];
    int pos_m = d.seg[1536 + warp];
    int kept = d.seg[2048 + warp];
    int m = 0;
    unsigned int lower = (1u << lane) - 1u;
#pragma unroll 4
    for (int base = warp * ppt; base < warp * ppt + ppt; base += 32) {
        int i = base + lane;
        bool in = i < warp * ppt + ppt;
        unsigned int q = in ? (unsigned int)(__ldg(grad + i) * (nb - 1) + 0.5f) : 0u;
        bool ia = in && q > thr, im = in && q == thr;
        unsigned int ab = __ballot_sync(0xffffffffu, ia);
        unsigned int me = __ballot_sync(0xffffffffu, im);
        if (ia) {
            int pos = pos_a + __popc(ab & lower);
            if (pos < P) d.sel_idx[pos] = i;
        }
        if (im) {
            int r = m + __popc(me & lower);
            if (r < kept) {
                int pos = pos_m + r;
                if (pos < P) d.sel_idx[pos] = i;
            }
        }
        pos_a += __popc(ab);
        m += __popc(me);
    }
}

// addVertexAttributesWithoutNormalsKernel3/4 (d2z.cu:700-936) and
// precomputeJacobian4Kernel (warp.cu:502-645), fused per selected point.
__global__ void k_attr_jac(const InstDesc *D, const int *active) {
    INST_DESC;
    if (!active[blockIdx.y]) return;
    int P = d.P, L = d.L, W = d.W, H = d.H, n = W * H;
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= P) return;
    int pix = d.sel_idx[k];
    float v[kVtxPlanes];
    vertex_record(d, pix, W, H, v);
    float p3x = v[0], p3y = v[1], p3z = v[2];
    float gx[kMaxLevels] = {0, 0, 0, 0}, gy[kMaxLevels] = {0, 0, 0, 0}, col[kMaxLevels] = {0, 0, 0, 0};
    gx[0] = v[5];
    gy[0] = v[6];
    col[0] = v[8];
    const float *T = d.calib + RC_TLR;
    const float *kc = d.calib + RC_KCR;
    const float *KR = d.calib + RC_KR;
    float rx, ry, rz;
    mul4(T, p3x, p3y, p3z, rx, ry, rz);
    {
        float pux = rx / rz, puy = ry / rz;
        float px, py;
        distort(pux, puy, kc, KR, px, py);
        if (in_bounds10(px, py, W, H)) {
            float a = 0.5f, b = -0.25f;
            float lx = px, ly = py;
            for (int l = 1; l < L; l++) {
                lx = a * lx + b;
                ly = a * ly + b;
                int wl = W >> l, hl = H >> l;
                int xdi = ftoi(lx), ydi = ftoi(ly);
                float fracX = lx - xdi, fracY = ly - ydi;
                const float *g = d.ref_gray[l];
                col[l] = bilin_clamped(xdi, ydi, fracX, fracY, wl, hl, g);
                float cN = bilin_clamped(xdi, ydi - 1, fracX, fracY, wl, hl, g);
                float cW = bilin_clamped(xdi - 1, ydi, fracX, fracY, wl, hl, g);
                float cE = bilin_clamped(xdi + 1, ydi, fracX, fracY, wl, hl, g);
                float cS = bilin_clamped(xdi, ydi + 1, fracX, fracY, wl, hl, g);
                gx[l] = (cE - cW) / 2.0f;
                gy[l] = (cS - cN) / 2.0f;
            }
        }
    }
    d.sel_xyz[k] = p3x;
    d.sel_xyz[P + k] = p3y;
    d.sel_xyz[2 * P + k] = p3z;
    for (int l = 0; l < L; l++) {
        d.sel_I[l][k] = col[l];
        if (d.sel_Ih[l]) d.sel_Ih[l][k] = __float2half_rn(col[l]);  // mixed precision
    }

    // precomputeJacobian4Kernel
    float optScaleIn = d.opt_in;
    rx *= optScaleIn;
    ry *= optScaleIn;
    rz *= optScaleIn;
    float dN0 = 1.0f / rz, dN1 = 0, dN2 = -rx / (rz * rz);
    float dN3 = 0, dN4 = 1.0f / rz, dN5 = -ry / (rz * rz);
    float x = rx / rz;
    float y = ry / rz;
    float x2 = x * x, y2 = y * y;
    float x4 = x2 * x2, y4 = y2 * y2;
    float r2 = x2 + y2, r4 = r2 * r2;
    float dD0 = 1 + kc[0] * (3 * x2 + y2) + kc[1] * (5 * x4 + 6 * x2 * y2 + y4) + kc[4] * r4 * (7 * x2 + y2);
    float dD1 = kc[0] * 2 * x * y + kc[1] * 4 * x * y * r2 + kc[4] * 6 * x * y * r4;
    float dD2 = kc[0] * 2 * y * x + kc[1] * 4 * x * y * r2 + kc[4] * 6 * x * y * r4;
    float dD3 = 1 + kc[0] * (3 * x2 + y2) + kc[1] * (5 * x4 + 6 * x2 * y2 + y4) + kc[4] * r4 * (7 * y2 + x2);
    const float dps[6][3] = {{0.0f, -rz, ry}, {rz, 0.0f, -rx}, {-ry, rx, 0.0f},
                             {1.0f, 0.0f, 0.0f}, {0.0f, 1.0f, 0.0f}, {0.0f, 0.0f, 1.0f}};
#pragma unroll
    for (int c = 0; c < 6; c++) {
        float drx, dry, drz;
        rot4(T, dps[c][0], dps[c][1], dps[c][2], drx, dry, drz);
        float dpnx = dN0 * drx + dN1 * dry + dN2 * drz;
        float dpny = dN3 * drx + dN4 * dry + dN5 * drz;
        float ddx = dD0 * dpnx + dD1 * dpny;
        float ddy = dD2 * dpnx + dD3 * dpny;
        float ddz = 0;
        float dp2x, dp2y, dp2z;
        mul3(KR, ddx, ddy, ddz, dp2x, dp2y, dp2z);
        for (int l = 0; l < L; l++) {
            float val;
            if (l == 0) val = dp2x * gx[0] + dp2y * gy[0];
            else {
                float s = (l == 1) ? 2.0f : (l == 2 ? 4.0f : 8.0f);
                val = (dp2x / s) * gx[l] + (dp2y / s) * gy[l];
            }
            d.sel_J[l][c * P + k] = val;
            if (d.sel_Jb[l]) d.sel_Jb[l][c * P + k] = __float2bfloat16_rn(val);  // mixed precision
        }
    }
}

// ------------------------------------------------------------------
// ICP: correspondence mask, compaction, Student-t weights
// ------------------------------------------------------------------

// (long long)x for 0 <= x < 2^63 (or x = -0) from the bits of x with integer
// operations: the float -> int64 conversion instruction issues on the FP64
// pipe, which is narrow on this GPU.
__device__ __forceinline__ long long trunc_f32_nonneg(float x) {
    uint32_t bits = __float_as_uint(x) & 0x7fffffffu;
    int E = (int)(bits >> 23);
    if (E < 127) return 0;  // x < 1
    uint64_t m = (uint64_t)((bits & 0x7fffffu) | 0x800000u);
    int sh = E - 150;
    return (long long)(sh >= 0 ? (m << sh) : (m >> -sh));
}

// the reference's int truncation of r^2 w (estimateVariance1024, rgb2gray.cu:519-521)
__device__ __forceinline__ long long trunc_prod(float r2, float w) {
    float prod = r2 * w;
    if (prod >= 0.0f && prod < 8388608.0f) return trunc_small(prod);
    return (prod >= 0.0f && prod < 9.0e18f) ? trunc_f32_nonneg(prod) : (prod >= 9.0e18f ? 9000000000000000000LL : 0);
}

// The Student-t weight (rgb2gray.cu:537-540; the first pass's sigma^2 is 100,
// rgb2gray.cu:827-850)
// by the reciprocal of sigma^2, which all pixels of a pass share, and the exact
// division of pair_math.cuh.  A squared residual below its range gives 5 + r^2 /
// sigma^2 = 5 by either division.
struct StudentW {
    float sigma2, y;
    bool plain;
    __device__ __forceinline__ explicit StudentW(float s2)
        : sigma2(s2), y(rcp_rn(s2)), plain(s2 >= 0x1p-20f && s2 <= 0x1p60f) {}
    // whether near() serves squared residuals of this sum (NaN does not)
    __device__ __forceinline__ bool in_range(float sum_r2) const { return plain && sum_r2 <= 0x1p40f; }
    __device__ __forceinline__ float near(float r2) const {
        float d = 5.0f + div_rn(r2, -sigma2, y);
        return div_rn(6.0f, -d, rcp_rn(d));
    }
    __device__ __forceinline__ float far(float r2) const { return ieee_div(6.0f, 5.0f + ieee_div(r2, sigma2)); }
    __device__ __forceinline__ float operator()(float r2) const { return in_range(r2) ? near(r2) : far(r2); }
    // the truncated products r^2 w of four pixels, added up; a pixel that is no
    // correspondence has r^2 = 0 and adds nothing
    __device__ __forceinline__ long long products(float4 r) const {
        if (in_range(((r.x + r.y) + r.z) + r.w)) {
            float a = r.x * near(r.x), b = r.y * near(r.y), c = r.z * near(r.z), e = r.w * near(r.w);
            if (fmaxf(fmaxf(a, b), fmaxf(c, e)) < 8388608.0f)
                return trunc_small(a) + trunc_small(b) + trunc_small(c) + trunc_small(e);
        }
        return trunc_prod(r.x, (*this)(r.x)) + trunc_prod(r.y, (*this)(r.y)) + trunc_prod(r.z, (*this)(r.z)) +
               trunc_prod(r.w, (*this)(r.w));
    }
};

// What the ICP kernels need of a level for every pixel: the current frame's
// points there and the projection into it.
struct IcpLevel {
    const float *z;     // level 0: the depth image (its points are formed from it)
    const float4 *cur;  // the other levels' points
    int w;
    float wm1, hm1, fx, cx, fy, cy, a, b, rfx, rfy;
    bool plain;  // the focal lengths are in the range of div_rn
    __device__ __forceinline__ IcpLevel(const InstDesc &d, int level) {
        w = d.W >> level;
        z = d.cur_z;
        cur = d.cur_pts[level];
        wm1 = (float)(w - 1);
        hm1 = (float)((d.H >> level) - 1);
        const float *K = d.calib + RC_KL;
        fx = K[0];
        cx = K[2];
        fy = K[4];
        cy = K[5];
        a = 1.0f / (float)(1 << level);
        b = 0.5f * (a - 1.0f);
        plain = div_in_range(fx, fy, fx);
        rfx = rcp_rn(fx);
        rfy = rcp_rn(fy);
    }
};

// The projection of the transformed point q into the level (icpResidualKernel2
// and icpResidualIndexKernel2, the reference's expressions without contraction:
// they decide which pixels count), with the exact division of pair_math.cuh.
// Returns whether it lies inside.
__device__ __forceinline__ bool icp_project(const IcpLevel &L, float qx, float qy, float qz, float &px, float &py) {
    float y = rcp_rn(qz), ux = div_rn(qx, -qz, y), uy = div_rn(qy, -qz, y);
    if (!div_in_range(qx, qy, qz)) {
        ux = ieee_div(qx, qz);
        uy = ieee_div(qy, qz);
    }
    px = L.a * (L.fx * ux + L.cx) + L.b;
    py = L.a * (L.fy * uy + L.cy) + L.b;
    return px >= 0.0f && px < L.wm1 && py >= 0.0f && py < L.hm1;
}

// The four taps of a projected pixel.  At level 0 they are depths, and the
// points are formed from them as genPointsCloud6Kernel does (d2z.cu:436-469; zero
// where there is no depth): a quarter of the bytes and of the cache lines that
// gathering points costs, for 36 operations, half of them packed.  (The division's
// operands are looked at from above only.  A numerator below its range, a depth or
// a distance from the principal point of less than 2^-60, still gives the rounded
// quotient down to 2^-102, then one within a unit in the last place, and a zero may
// lose its sign: nothing in a sum of millimetres.)  At the other
// levels (averages of points) they are float4 points.
template <bool kDepth> struct IcpTaps;
template <> struct IcpTaps<true> {
    float z[4];
    __device__ __forceinline__ void load(const IcpLevel &L, int o) {
        const float *p = L.z + o, *q = p + L.w;
        z[0] = __ldg(p);
        z[1] = __ldg(p + 1);
        z[2] = __ldg(q);
        z[3] = __ldg(q + 1);
    }
    // which taps have a point
    __device__ __forceinline__ bool first() const { return z[0] < 0.0f; }
    __device__ __forceinline__ bool all() const { return z[0] < 0.0f && z[1] < 0.0f && z[2] < 0.0f && z[3] < 0.0f; }
    __device__ __forceinline__ void points(const IcpLevel &L, float xf, float yf, float *x, float *y, float *zc) const {
#pragma unroll
        for (int k = 0; k < 4; k++) zc[k] = fminf(z[k], 0.0f);  // a positive depth or NaN has no point
        float2 X = make_float2(xf - L.cx, (xf + 1.0f) - L.cx);
        float Y0 = yf - L.cy, Y1 = (yf + 1.0f) - L.cy;
        float2 z0 = make_float2(zc[0], zc[1]), z1 = make_float2(zc[2], zc[3]);
        float2 ax = mul2(X, z0), bx = mul2(X, z1), ay = mul2(dup2(Y0), z0), by = mul2(dup2(Y1), z1);
        float2 nfx = dup2(-L.fx), rx = dup2(L.rfx), nfy = dup2(-L.fy), ry = dup2(L.rfy);
        float2 qx = div_rn2(ax, nfx, rx), sx = div_rn2(bx, nfx, rx), qy = div_rn2(ay, nfy, ry), sy = div_rn2(by, nfy, ry);
        if (!L.plain || !(fminf(fminf(zc[0], zc[1]), fminf(zc[2], zc[3])) >= -1e12f)) {
            qx = make_float2(ieee_div(ax.x, L.fx), ieee_div(ax.y, L.fx));
            sx = make_float2(ieee_div(bx.x, L.fx), ieee_div(bx.y, L.fx));
            qy = make_float2(ieee_div(ay.x, L.fy), ieee_div(ay.y, L.fy));
            sy = make_float2(ieee_div(by.x, L.fy), ieee_div(by.y, L.fy));
        }
        x[0] = qx.x; x[1] = qx.y; x[2] = sx.x; x[3] = sx.y;
        y[0] = qy.x; y[1] = qy.y; y[2] = sy.x; y[3] = sy.y;
    }
};
template <> struct IcpTaps<false> {
    float4 t[4];
    __device__ __forceinline__ void load(const IcpLevel &L, int o) {
        const float4 *p = L.cur + o, *q = p + L.w;
        t[0] = __ldg(p);
        t[1] = __ldg(p + 1);
        t[2] = __ldg(q);
        t[3] = __ldg(q + 1);
    }
    __device__ __forceinline__ bool first() const { return t[0].w != 0.0f; }
    __device__ __forceinline__ bool all() const {
        return t[0].w != 0.0f && t[1].w != 0.0f && t[2].w != 0.0f && t[3].w != 0.0f;
    }
    __device__ __forceinline__ void points(const IcpLevel &, float, float, float *x, float *y, float *z) const {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            x[k] = t[k].x;
            y[k] = t[k].y;
            z[k] = t[k].z;
        }
    }
};

// bilinearInterpolation6 of the taps at the projection (px, py), kernelUtils.h:305-316
template <bool kDepth>
__device__ __forceinline__ void icp_blend(const IcpLevel &L, const IcpTaps<kDepth> &t, float px, float py, float &cx,
                                          float &cy, float &cz) {
    // trunc by a sum rounded toward zero (index_sum): no conversions
    float xf = index_sum(px) - 8388608.0f, yf = index_sum(py) - 8388608.0f;
    float u = px - xf, v = py - yf;
    float x[4], y[4], z[4];
    t.points(L, xf, yf, x, y, z);
    float w0 = (1 - u) * (1 - v), w1 = u * (1 - v), w2 = (1 - u) * v, w3 = u * v;
    cx = w0 * x[0] + w1 * x[1] + w2 * x[2] + w3 * x[3];
    cy = w0 * y[0] + w1 * y[1] + w2 * y[2] + w3 * y[3];
    cz = w0 * z[0] + w1 * z[1] + w2 * z[2] + w3 * z[3];
}

__device__ __forceinline__ int icp_tap_index(const IcpLevel &L, bool inside, float px, float py) {
    return inside ? index_of(index_sum(px)) + index_of(index_sum(py)) * L.w : 0;
}

// The mask and squared residual of a pixel of the level (icpResidualKernel2) from
// its reference point (x y z, z NaN where there is none) and normal.
template <bool kDepth>
__device__ __forceinline__ bool icp_mask_pixel(const IcpLevel &L, const float *T, const float *p, float &r2) {
    r2 = 0.0f;
    if (p[2] != p[2]) return false;
    float qx, qy, qz, px, py, nx, ny, nz, cx, cy, cz;
    mul4(T, p[0], p[1], p[2], qx, qy, qz);
    if (!icp_project(L, qx, qy, qz, px, py)) return false;
    IcpTaps<kDepth> t;
    t.load(L, icp_tap_index(L, true, px, py));
    if (!t.all()) return false;
    rot4(T, p[3], p[4], p[5], nx, ny, nz);
    icp_blend<kDepth>(L, t, px, py, cx, cy, cz);
    float res = (cx - qx) * nx + (cy - qy) * ny + (cz - qz) * nz;
    r2 = res * res;
    return true;
}

// Whether this CTA is the last of the instance's `nblk` CTAs of the launch to
// finish its partial total (written by thread 0 before the call): thread 0 makes
// the total visible, then takes a ticket from the instance's counter; the CTA
// holding the last ticket resets the counter for the next launch and may read
// every partial total.  No CTA waits for another.
__device__ __forceinline__ bool icp_last_block(const InstDesc &d, int nblk) {
    __shared__ int s_last;
    if (threadIdx.x == 0) {
        __threadfence();
        unsigned int k = atomicAdd(d.counter + 1, 1u);
        s_last = (k == (unsigned int)nblk - 1u);
        if (s_last) {
            atomicExch(d.counter + 1, 0u);
            __threadfence();
        }
    }
    __syncthreads();
    return s_last != 0;
}

// Blocks [b0, b1) of 1024 pixels, four per thread, kBatch at a time: a batch's
// taps are in flight together, and meanwhile the next batch's points and normals.
template <bool kDepth>
__device__ __forceinline__ void icp_mask_blocks(const InstDesc &d, int level, const float *T, int b0, int b1, int n,
                                                int &cnt, long long &vsum) {
    constexpr int kBatch = kDepth ? 2 : 1;
    const IcpLevel L(d, level);
    const StudentW first(100.0f);
    const float *pl = d.ref_pl[level] + (size_t)b0 * 6 * kChunk + threadIdx.x;
    float next[kBatch][6];
#pragma unroll
    for (int u = 0; u < kBatch; u++)
#pragma unroll
        for (int k = 0; k < 6; k++) next[u][k] = __ldg(pl + k * kChunk + u * kLanes);
    for (int b = b0; b < b1; b++, pl += 6 * kChunk) {
        int i = b * kChunk + threadIdx.x;
        float r4[4];
#pragma unroll
        for (int g = 0; g < 4; g += kBatch) {
            // (past the last pixel the planes hold no point: nothing is stored)
            float p[kBatch][6], q[kBatch][3], px[kBatch], py[kBatch];
            bool in[kBatch];
            IcpTaps<kDepth> tap[kBatch];
#pragma unroll
            for (int u = 0; u < kBatch; u++) {
#pragma unroll
                for (int k = 0; k < 6; k++) p[u][k] = next[u][k];
                mul4(T, p[u][0], p[u][1], p[u][2], q[u][0], q[u][1], q[u][2]);
                in[u] = p[u][2] == p[u][2] && i + (g + u) * kLanes < n && icp_project(L, q[u][0], q[u][1], q[u][2], px[u], py[u]);
                tap[u].load(L, icp_tap_index(L, in[u], px[u], py[u]));
            }
            if (g + kBatch < 4 || b + 1 < b1) {
                const float *nx = g + kBatch < 4 ? pl + (g + kBatch) * kLanes : pl + 6 * kChunk;
#pragma unroll
                for (int u = 0; u < kBatch; u++)
#pragma unroll
                    for (int k = 0; k < 6; k++) next[u][k] = __ldg(nx + k * kChunk + u * kLanes);
            }
#pragma unroll
            for (int u = 0; u < kBatch; u++) {
                float nx, ny, nz, cx, cy, cz;
                bool ok = in[u] && tap[u].all();
                float r2 = 0.0f;
                if (ok) {
                    rot4(T, p[u][3], p[u][4], p[u][5], nx, ny, nz);
                    icp_blend<kDepth>(L, tap[u], px[u], py[u], cx, cy, cz);
                    float res = (cx - q[u][0]) * nx + (cy - q[u][1]) * ny + (cz - q[u][2]) * nz;
                    r2 = res * res;
                }
                int at = i + (g + u) * kLanes;
                if (at < n) {
                    d.icp_r2[at] = r2;
                    d.icp_mask[at] = ok;
                }
                r4[g + u] = r2;
                cnt += ok;
            }
        }
        vsum += first.products(make_float4(r4[0], r4[1], r4[2], r4[3]));
    }
}

// icpResidualKernel2 (rgb2gray.cu:223-260) with initWeightsKernel's first
// Student-t weight (rgb2gray.cu:827-850): per pixel of the level, whether it is
// a correspondence at the level's start pose and its squared residual; per
// block of 1024 pixels the number of correspondences and the exact int64 sum
// of the truncated r^2 w0 products (the first variance sum).  The ICP sums of
// the iterations run over the pixel grid, so no compacted list is built.
// What bounds it is the latency of its two round trips per pixel (33 bytes of
// DRAM traffic each at level 0: 3.4 TB/s), so a CTA takes blocks_per_cta blocks
// in turn with the next pixels' points and normals on their way while these are
// evaluated: level 0 of 30 640x480 instances 90 us against 105 us with a block
// per CTA and one pixel after another, level 1 29 against 34.  More pixels at
// once in fewer CTAs (4 pixels, 2 per SM: 103 us) or the other way round (1
// pixel, 6 per SM: 94) is no better, nor are L2 prefetches of the next block.
__global__ void __launch_bounds__(kLanes, kMaskCtas)
    k_icp_mask(const InstDesc *D, int level, int blocks_per_cta) {
    pdl_trigger();
    __shared__ InstDesc sd;
    __shared__ float sT[16];
    __shared__ int s_cnt[kLanes / 32];
    __shared__ long long s_var[kLanes / 32];
    load_desc(sd, D + blockIdx.y);
    __syncthreads();
    const InstDesc &d = sd;
    if (level >= d.L || d.mode == RECON_PHOTOMETRIC) return;
    if (d.iters[d.L - 1 - level] <= 0) return;
    int n = (d.W >> level) * (d.H >> level);
    // the grid covers the batch's largest level; this instance has fewer blocks
    // (its per-block arrays hold exactly that many entries)
    int nblk = (n + kChunk - 1) / kChunk;
    int b0 = blockIdx.x * blocks_per_cta, b1 = min(b0 + blocks_per_cta, nblk);
    if (b0 >= nblk) return;
    pdl_wait();
    if (threadIdx.x < 16) sT[threadIdx.x] = __ldcg(d.T + threadIdx.x);
    if (blockIdx.x == 0 && threadIdx.x == 0) d.work[2] += (unsigned long long)n;
    __syncthreads();
    int cnt = 0;
    long long vsum = 0;
    if (level == 0) icp_mask_blocks<true>(d, level, sT, b0, b1, n, cnt, vsum);
    else icp_mask_blocks<false>(d, level, sT, b0, b1, n, cnt, vsum);
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    for (int o = 16; o > 0; o >>= 1) vsum += __shfl_xor_sync(0xffffffffu, vsum, o);
    int wid = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        s_cnt[wid] = cnt;
        s_var[wid] = vsum;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int c = 0;
        long long v = 0;
        for (int k = 0; k < kLanes / 32; k++) {
            c += s_cnt[k];
            v += s_var[k];
        }
        // the total of the CTA's blocks is its first block's
        for (int b = b0; b < b1; b++) {
            d.icp_blkcnt[b] = b == b0 ? c : 0;
            d.icp_blkvar[b] = b == b0 ? v : 0;
        }
    }
}

// Student-t pass `pass` (1..3) of a level (updateWeightsKernel /
// clampWeightsKernel, rgb2gray.cu:549-569) over the level's pixel grid: CTA x
// of instance blockIdx.y takes the 1024-pixel blocks [x K, (x+1) K) of the
// instance, K = blocks_per_cta (about one wave of CTAs over the batch), a
// thread four consecutive pixels of each block with the loads of four blocks
// in flight.  Every correspondence is weighed with the variance of the
// previous pass; passes 1 and 2 add the truncated products r^2 w into the
// CTA's partial sum (icp_part) and the instance's last CTA forms the total
// icp_var[pass]; pass 3 clamps at 1 and writes every pixel's weight (0 where
// the pixel is not a correspondence).  Pass 1 first adds up k_icp_mask's block
// totals (every CTA, from L2): the correspondence count and the first
// variance sum, which CTA 0 stores.  The sums are exact int64 sums, so the
// result does not depend on how the pixels are split; one launch per pass
// keeps every SM busy without any CTA waiting on another.  48 registers: five
// CTAs per SM (kPassCtaSlots).  The three passes of
// level 0 of 30 640x480 instances take 45 us, level 1 23; 63 and 27 with IEEE
// divisions in place of those by a reciprocal (StudentW).
// Passes 1 and 2 need no mask: a pixel that is no correspondence has r^2 = 0.
__global__ void __launch_bounds__(kLanes, 5) k_icp_student_pass(const InstDesc *D, int level, int pass,
                                                             int blocks_per_cta) {
    pdl_trigger();
    __shared__ InstDesc sd;
    __shared__ long long s_var[kLanes / 32];
    __shared__ int s_cnt[kLanes / 32];
    load_desc(sd, D + blockIdx.y);
    __syncthreads();
    const InstDesc &d = sd;
    if (level >= d.L || d.mode == RECON_PHOTOMETRIC) return;
    if (d.iters[d.L - 1 - level] <= 0) return;
    int n = (d.W >> level) * (d.H >> level);
    int nblk = (n + kChunk - 1) / kChunk;
    int nctas = (nblk + blocks_per_cta - 1) / blocks_per_cta;
    if ((int)blockIdx.x >= nctas) return;
    int b_first = blockIdx.x * blocks_per_cta;
    int b_last = min(b_first + blocks_per_cta, nblk);
    int wid = threadIdx.x >> 5;
    pdl_wait();
    int nsel;
    long long var;
    if (pass == 1) {
        int c = 0;
        long long v = 0;
        for (int k = threadIdx.x; k < nblk; k += kLanes) {
            c += __ldcg(d.icp_blkcnt + k);
            v += __ldcg(d.icp_blkvar + k);
        }
        c = __reduce_add_sync(0xffffffffu, c);
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0) {
            s_cnt[wid] = c;
            s_var[wid] = v;
        }
        __syncthreads();
        nsel = 0;
        var = 0;
        for (int k = 0; k < kLanes / 32; k++) {
            nsel += s_cnt[k];
            var += s_var[k];
        }
        __syncthreads();  // s_var is reused for this pass's sum
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            d.icp_nsel[level] = nsel;
            // ICP weight of the fused system, kept off the iteration's critical path
            d.fuse_c2[level] = (double)d.lambda / (double)nsel;
            d.icp_var[0] = (unsigned long long)var;
        }
    } else {
        nsel = __ldcg(d.icp_nsel + level);
        var = (long long)__ldcg(d.icp_var + pass - 1);
    }
    float Sf = (float)var;
    float minVal = (float)nsel;
    float vv = (nsel <= 1024) ? Sf : (Sf < minVal ? minVal : Sf);
    const StudentW weight(vv / (float)nsel);
    long long vsum = 0;
    for (int b0 = b_first; b0 < b_last; b0 += 4) {
        float4 r[4];
        uchar4 m[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            int i = (b0 + u) * kChunk + 4 * threadIdx.x;
            r[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            m[u] = make_uchar4(0, 0, 0, 0);
            if (b0 + u >= b_last || i >= n) continue;
            if (i + 3 < n) {
                // 16- and 4-byte aligned: the arrays start on 256-byte boundaries
                r[u] = __ldcg(reinterpret_cast<const float4 *>(d.icp_r2 + i));
                if (pass == 3) m[u] = __ldcg(reinterpret_cast<const uchar4 *>(d.icp_mask + i));
            } else {
                // the instance's last pixels (n not a multiple of 4)
                r[u].x = __ldcg(d.icp_r2 + i);
                m[u].x = __ldcg(d.icp_mask + i);
                if (i + 1 < n) {
                    r[u].y = __ldcg(d.icp_r2 + i + 1);
                    m[u].y = __ldcg(d.icp_mask + i + 1);
                }
                if (i + 2 < n) {
                    r[u].z = __ldcg(d.icp_r2 + i + 2);
                    m[u].z = __ldcg(d.icp_mask + i + 2);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            int i = (b0 + u) * kChunk + 4 * threadIdx.x;
            if (b0 + u >= b_last) continue;
            if (pass == 3) {
                // pixels past the level's last one have mask 0: the weights
                // are zero up to the end of the block
                float4 w;
                if (weight.in_range(((r[u].x + r[u].y) + r[u].z) + r[u].w))
                    w = make_float4(weight.near(r[u].x), weight.near(r[u].y), weight.near(r[u].z), weight.near(r[u].w));
                else
                    w = make_float4(weight(r[u].x), weight(r[u].y), weight(r[u].z), weight(r[u].w));
                w.x = m[u].x ? fminf(w.x, 1.0f) : 0.0f;
                w.y = m[u].y ? fminf(w.y, 1.0f) : 0.0f;
                w.z = m[u].z ? fminf(w.z, 1.0f) : 0.0f;
                w.w = m[u].w ? fminf(w.w, 1.0f) : 0.0f;
                *reinterpret_cast<float4 *>(d.icp_w + i) = w;
            } else {
                vsum += weight.products(r[u]);
            }
        }
    }
    if (pass == 3) return;
    for (int o = 16; o > 0; o >>= 1) vsum += __shfl_xor_sync(0xffffffffu, vsum, o);
    if ((threadIdx.x & 31) == 0) s_var[wid] = vsum;
    __syncthreads();
    if (threadIdx.x == 0) {
        long long v = 0;
        for (int k = 0; k < kLanes / 32; k++) v += s_var[k];
        d.icp_part[blockIdx.x] = v;
    }
    if (!icp_last_block(d, nctas)) return;
    long long v = 0;
    for (int k = threadIdx.x; k < nctas; k += kLanes) v += __ldcg(d.icp_part + k);
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) s_var[wid] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        long long tot = 0;
        for (int k = 0; k < kLanes / 32; k++) tot += s_var[k];
        d.icp_var[pass] = (unsigned long long)tot;
    }
}

// ------------------------------------------------------------------
// one Gauss-Newton iteration for every instance
// ------------------------------------------------------------------

constexpr int kIterThreads = kIterBlock;  // one canonical lane (4 points of a chunk) per thread
constexpr int kCluster = kIterCluster;
constexpr int kFxTerms = 27 * kFxLimbs;

// Constants of photo_pair, alike in both halves: the pose, the rig's transforms
// (their upper three rows), the RGB camera with its distortion, the level's
// scale and offset, the IR camera's upper two rows.
struct alignas(16) PhotoConsts {
    float2 T[12], TLR[12], TRL[12], KR[4], kc[3], ab[2], KL[6];
    __device__ __forceinline__ void set_level(const InstDesc &d, int level) {
        int t = threadIdx.x;
        float s = 1.0f / (float)(1 << level);
        if (t < 12) {
            TLR[t] = dup2(d.calib[RC_TLR + t]);
            TRL[t] = dup2(d.calib[RC_TRL + t]);
        }
        if (t < 6) KL[t] = dup2(d.calib[RC_KL + t]);
        if (t < 3) kc[t] = dup2(d.calib[RC_KCR + (t < 2 ? t : 4)]);
        if (t < 4) KR[t] = dup2(d.calib[RC_KR + (t < 2 ? 2 * t : t + 2)]);  // entries 0, 2, 4, 5
        if (t < 2) ab[t] = dup2(t == 0 ? s : 0.5f * (s - 1.0f));
    }
    __device__ __forceinline__ void set_pose(float v) {
        if (threadIdx.x < 12) T[threadIdx.x] = dup2(v);
    }
};

// 16-byte aligned: stage is the destination of 16-byte cp.async copies
struct alignas(16) IterShared {
    // ICP: the terms of the chunk being reduced (term k of pixel i at
    // 1024 k + i); photometric: the Jacobian of the CTA's first chunk.  Once a warp
    // has read its points, the 28 runs of 32 floats they occupied are its own
    // scratch for the reduction (warp_terms).
    float stage[7 * kChunk];
    union {
        uint4 sums[kIterBlock / 32][27];  // the warps' fixed-point sums, when the CTA is done
        int peers[kCluster][256];         // before: the histograms of the cluster's CTAs, written by them
    };
    PhotoConsts photo;
    float T[16];
    int bad;        // an accumulated value was out of range
    int hist[256];  // this CTA's photometric histogram
    int median;
    int warp_tot[kIterBlock / 32];
};

// The allocation-free entry point's single CTA.
struct PhotoShared {
    float T[16];
    long long fx[27][kFxLimbs];  // fixed-point sums of the warp totals
    int fx_bad;
    double A_ph[27];
    int hist[256];
    int median;
    SolveScratch S;
};

struct SolveShared {
    float T[16];
    double A_icp[27];
    SolveScratch S;
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory"); }

// address of `p` (a shared-memory variable of this CTA) in CTA `rank` of the cluster
template <class T> __device__ __forceinline__ T *cluster_peer(T *p, int rank) {
    unsigned long long out;
    asm volatile("mapa.u64 %0, %1, %2;\n" : "=l"(out) : "l"((unsigned long long)p), "r"(rank));
    return reinterpret_cast<T *>(out);
}

// Adds warp total v of term q to the sums of the allocation-free entry
// point's CTA; its 8 warps add to the same limbs with shared-memory atomics.
__device__ __forceinline__ void fx_add_term(PhotoShared &sh, int q, float v) {
    int k0, bad = 0;
    long long lo, hi;
    fx_split(v, k0, lo, hi, bad);
    if (lo) atomicAdd(reinterpret_cast<unsigned long long *>(&sh.fx[q][k0]), (unsigned long long)lo);
    if (hi) atomicAdd(reinterpret_cast<unsigned long long *>(&sh.fx[q][k0 + 1]), (unsigned long long)hi);
    if (bad) sh.fx_bad = 1;
}

// Adds the CTA's sums, a 128-bit value per warp and term (lane q of a warp:
// term q), to the instance's limbs: the warps' words are added as limbs, the top
// one signed, so no carries are needed.  sh.bad must be 0 before.
__device__ __forceinline__ void fx_flush(IterShared &sh, const uint32_t *acc, int bad, unsigned long long *dst,
                                         int *dst_bad) {
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane < 27) sh.sums[w][lane] = make_uint4(acc[0], acc[1], acc[2], acc[3]);
    if (lane < 27 && bad) sh.bad = 1;
    __syncthreads();
    if (threadIdx.x < kFxTerms) {
        const uint32_t *words = reinterpret_cast<const uint32_t *>(&sh.sums[0][0]) + threadIdx.x;
        long long v = 0;
#pragma unroll
        for (int k = 0; k < kIterBlock / 32; k++) {
            uint32_t x = words[k * kFxTerms];
            v += (threadIdx.x & 3) == 3 ? (long long)(int)x : (long long)x;
        }
        if (v) atomicAdd(dst + threadIdx.x, (unsigned long long)v);
    }
    if (threadIdx.x == 0 && sh.bad) atomicOr(dst_bad, 1);
}

// canonical per-lane accumulation of the 27 normal-equation terms, one fused
// multiply-add per product (the oracle's fmaf)
__device__ __forceinline__ void acc27(float *s, const float *j, float r) {
    int q = 0;
#pragma unroll
    for (int a = 0; a < 6; a++)
#pragma unroll
        for (int c = a; c < 6; c++, q++) s[q] = __fmaf_rn(j[a], j[c], s[q]);
#pragma unroll
    for (int c = 0; c < 6; c++, q++) s[q] = __fmaf_rn(j[c], r, s[q]);
}

// The same 27 sums two by two: 12 packed and 3 plain multiply-adds, each half
// rounded as the plain one is, for 27.  The ICP term's pixels leave their terms as
// pairs, 8 shared-memory accesses a pixel for 14: 30 segments 14538 -> 14337 us.
// (The photometric term, whose Jacobian comes by columns, is 1% slower so.)
struct Terms27 {
    float2 p[12];
    float s[3];
    __device__ __forceinline__ Terms27() {
#pragma unroll
        for (int k = 0; k < 12; k++) p[k] = make_float2(0.0f, 0.0f);
        s[0] = s[1] = s[2] = 0.0f;
    }
    __device__ __forceinline__ void add(float2 a, float2 b, float2 c, float r) {
        p[0] = fma2(dup2(a.x), a, p[0]);
        p[1] = fma2(dup2(a.x), b, p[1]);
        p[2] = fma2(dup2(a.x), c, p[2]);
        s[0] = __fmaf_rn(a.y, a.y, s[0]);
        p[3] = fma2(dup2(a.y), b, p[3]);
        p[4] = fma2(dup2(a.y), c, p[4]);
        p[5] = fma2(dup2(b.x), b, p[5]);
        p[6] = fma2(dup2(b.x), c, p[6]);
        s[1] = __fmaf_rn(b.y, b.y, s[1]);
        p[7] = fma2(dup2(b.y), c, p[7]);
        p[8] = fma2(dup2(c.x), c, p[8]);
        s[2] = __fmaf_rn(c.y, c.y, s[2]);
        p[9] = fma2(dup2(r), a, p[9]);
        p[10] = fma2(dup2(r), b, p[10]);
        p[11] = fma2(dup2(r), c, p[11]);
    }
    // in acc27's order
    __device__ __forceinline__ void terms(float *v) const {
        const float t[27] = {p[0].x, p[0].y, p[1].x, p[1].y, p[2].x, p[2].y, s[0],   p[3].x,  p[3].y,
                             p[4].x, p[4].y, p[5].x, p[5].y, p[6].x, p[6].y, s[1],   p[7].x,  p[7].y,
                             p[8].x, p[8].y, s[2],   p[9].x, p[9].y, p[10].x, p[10].y, p[11].x, p[11].y};
#pragma unroll
        for (int k = 0; k < 27; k++) v[k] = t[k];
    }
};

// Warp totals of the 27 terms by recursive halving: at the step with offset o
// each lane keeps half of its values and adds the partner's copy of them, so
// lane q ends with term q.  Every addition pairs the same two partial sums as
// the canonical xor butterfly (offsets 16, 8, 4, 2, 1), so the totals are the
// butterfly's bit for bit, with 31 shuffles instead of 135.
__device__ __forceinline__ float warp_terms(const float *v) {
    int lane = threadIdx.x & 31;
    float a[16];
    bool h = lane & 16;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        float x = v[i], y = (i + 16 < 27) ? v[i + 16] : 0.0f;
        float send = h ? x : y, keep = h ? y : x;
        a[i] = keep + __shfl_xor_sync(kFull, send, 16);
    }
    float b[8];
    h = lane & 8;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        float send = h ? a[i] : a[i + 8], keep = h ? a[i + 8] : a[i];
        b[i] = keep + __shfl_xor_sync(kFull, send, 8);
    }
    float c[4];
    h = lane & 4;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        float send = h ? b[i] : b[i + 4], keep = h ? b[i + 4] : b[i];
        c[i] = keep + __shfl_xor_sync(kFull, send, 4);
    }
    float e[2];
    h = lane & 2;
#pragma unroll
    for (int i = 0; i < 2; i++) {
        float send = h ? c[i] : c[i + 2], keep = h ? c[i + 2] : c[i];
        e[i] = keep + __shfl_xor_sync(kFull, send, 2);
    }
    h = lane & 1;
    float send = h ? e[0] : e[1], keep = h ? e[1] : e[0];
    return keep + __shfl_xor_sync(kFull, send, 1);
}

// The same totals through shared memory: `own` points to the warp's first run
// of 32 floats, run r = 4 k + m lies 1024 k + 256 m floats on (all lanes past
// their last use of them).  Run q takes the lanes' term q, rotated by 4q so that
// neither the stores nor the 16-byte loads of 8 runs at once meet in a bank, and
// lane q adds the butterfly's pairs of run q two at a time.  51 instructions
// where the recursive halving takes 124 (31 shuffles of 4 issue cycles each
// among them).  Returns term q on lane q < 27; the runs may be written again
// after the call.
__device__ __forceinline__ float warp_terms(const float *v, float *own) {
    int lane = threadIdx.x & 31;
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 27; q++) own[(q >> 2) * kChunk + (q & 3) * kLanes + ((lane + 4 * q) & 31)] = v[q];
    __syncwarp();
    int q = lane < 27 ? lane : 26;
    const float *run = own + (q >> 2) * kChunk + (q & 3) * kLanes;
    float2 s[8];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        float4 x = *reinterpret_cast<const float4 *>(run + ((4 * i + 4 * q) & 31));
        float4 y = *reinterpret_cast<const float4 *>(run + ((16 + 4 * i + 4 * q) & 31));
        s[2 * i] = plus2(make_float2(x.x, x.y), make_float2(y.x, y.y));  // lanes l and l ^ 16
        s[2 * i + 1] = plus2(make_float2(x.z, x.w), make_float2(y.z, y.w));
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 4; i++) s[i] = plus2(s[i], s[i + 4]);  // l ^ 8
    s[0] = plus2(s[0], s[2]);                                  // l ^ 4
    s[1] = plus2(s[1], s[3]);
    s[0] = plus2(s[0], s[1]);                                  // l ^ 2
    return s[0].x + s[0].y;                                    // l ^ 1
}

// Median bin of an instance histogram (seekThreshold64Kernel,
// histogram64.cu:48-61): first bin whose cumulative count exceeds P/2.  Warp 0.
template <class Shared>
__device__ __forceinline__ void hist_median(Shared &sh, const int *hist, int nb, int P) {
    if (threadIdx.x >= 32) return;
    int lane = threadIdx.x;
    int per = (nb + 31) / 32;
    int loc = 0;
    for (int k = 0; k < per; k++) {
        int bin = lane * per + k;
        if (bin < nb) loc += hist[bin];
    }
    int incl = loc;
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    int half = P / 2;
    unsigned int over = __ballot_sync(0xffffffffu, incl > half);
    if (over) {
        int l0 = __ffs(over) - 1;
        if (lane == l0) {
            int acc = incl - loc, med = 0;
            for (int k = 0; k < per; k++) {
                int bin = lane * per + k;
                if (bin < nb) {
                    acc += hist[bin];
                    if (acc > half) { med = bin; break; }
                }
            }
            sh.median = med;
        }
    } else if (lane == 0) {
        sh.median = 0;
    }
}

// One photometric iteration by a single 256-thread CTA (the allocation-free
// entry point): residuals, histogram, median, weights and the fixed-point sums
// of all P points; the 27 terms end in sh.A_ph.
__device__ void photo_iteration(const InstDesc &d, PhotoShared &sh, int level) {
    int P = d.P;
    int w = d.W >> level, h = d.H >> level;
    float a = 1.0f / (float)(1 << level);
    float b = 0.5f * (a - 1.0f);
    const float *img = d.cur_gray[level];
    const float *I = d.sel_I[level];
    int nb = d.hist_bins;
    for (int k = threadIdx.x; k < nb; k += blockDim.x) sh.hist[k] = 0;
    for (int k = threadIdx.x; k < kFxTerms; k += blockDim.x) (&sh.fx[0][0])[k] = 0;
    if (threadIdx.x == 0) sh.fx_bad = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < P; i += blockDim.x) {
        float r, zw;
        photo_residual(d.calib, sh.T, a, b, d.sel_xyz[i], d.sel_xyz[P + i], d.sel_xyz[2 * P + i], I[i], img, w, h,
                       d.cur_z, d.W, d.H, r, zw);
        d.ph_r[i] = r;
        d.ph_zw[i] = zw;
        atomicAdd(&sh.hist[mad_bin(r, nb)], 1);
    }
    __syncthreads();
    hist_median(sh, sh.hist, nb, P);
    __syncthreads();
    float s = mad_scale(sh.median, nb);
    const float *J = d.sel_J[level];
    int t = threadIdx.x, lane = t & 31;
    for (int c = 0; c < P / kChunk; c++) {
        float acc[27];
#pragma unroll
        for (int q = 0; q < 27; q++) acc[q] = 0.0f;
        for (int m = 0; m < 4; m++) {
            int i = c * kChunk + t + kLanes * m;
            float r = d.ph_r[i];
            float wv = tukey_weight(r, d.ph_zw[i], s);
            float jw[6];
#pragma unroll
            for (int k = 0; k < 6; k++) jw[k] = J[k * P + i] * wv;
            acc27(acc, jw, r * wv);
        }
        float v = warp_terms(acc);
        if (lane < 27) fx_add_term(sh, lane, v);
    }
    __syncthreads();
    if (threadIdx.x < 27) {
        long long L[kFxLimbs];
#pragma unroll
        for (int k = 0; k < kFxLimbs; k++) L[k] = sh.fx[threadIdx.x][k];
        sh.A_ph[threadIdx.x] = sh.fx_bad ? __longlong_as_double(0x7ff8000000000000LL) : fx_to_double(L);
    }
}

// icpResidualIndexKernel2, rgb2gray.cu:323-390, for one pixel of the level from
// its reference point p, normal n and weight, its transformed point q, the
// projection (px, py) of q and the taps there; inside: the pixel has a weight
// and q projects into the level (else, as in the reference, zeros).  The rotated
// normal, the residual and the Jacobian, continuous terms of the normal equations
// only, are evaluated with fused multiply-adds (one rounding per multiply-add;
// the oracle's orc_icp_residual_jacobian_grid states the same sequence with fmaf).
template <bool kDepth>
__device__ __forceinline__ void icp_point(const IcpLevel &L, const float *T, float opt_in, float weight, const float *p,
                                          const float *n, const float *q, float px, float py, bool inside,
                                          const IcpTaps<kDepth> &t, float *j, float &res) {
    res = 0.0f;
#pragma unroll
    for (int c = 0; c < 6; c++) j[c] = 0.0f;
    float cx, cy, cz;
    if (!(inside && t.first())) return;
    icp_blend<kDepth>(L, t, px, py, cx, cy, cz);
    if (!(fabsf(cz - q[2]) < 300.0f)) return;
    float mx = __fmaf_rn(T[2], n[2], __fmaf_rn(T[1], n[1], T[0] * n[0]));
    float my = __fmaf_rn(T[6], n[2], __fmaf_rn(T[5], n[1], T[4] * n[0]));
    float mz = __fmaf_rn(T[10], n[2], __fmaf_rn(T[9], n[1], T[8] * n[0]));
    float rx = cx - q[0], ry = cy - q[1], rz = cz - q[2];
    res = opt_in * weight * __fmaf_rn(rz, mz, __fmaf_rn(ry, my, rx * mx));
    // The reference rotates the columns of [p]x and [n]x and the unit vectors
    // with full 3x3 products.  The terms it multiplies by an exact 0 or 1 are
    // dropped here: for a finite pose that changes at most the sign of a zero
    // Jacobian entry, and signed zeros add nothing to the fixed-point sums.
    // A row: -m . b + r . c with b = T_a p_a + T_b p_b, c likewise of n
    auto row = [&](int a, float pa, float na, int b, float pb, float nb) {
        float s = -mx * __fmaf_rn(T[a], pa, T[b] * pb);
        s = __fmaf_rn(-my, __fmaf_rn(T[4 + a], pa, T[4 + b] * pb), s);
        s = __fmaf_rn(-mz, __fmaf_rn(T[8 + a], pa, T[8 + b] * pb), s);
        s = __fmaf_rn(rx, __fmaf_rn(T[a], na, T[b] * nb), s);
        s = __fmaf_rn(ry, __fmaf_rn(T[4 + a], na, T[4 + b] * nb), s);
        return __fmaf_rn(rz, __fmaf_rn(T[8 + a], na, T[8 + b] * nb), s);
    };
    float so = -opt_in * weight;
    j[0] = so * row(1, -p[2], -n[2], 2, p[1], n[1]);
    j[1] = so * row(0, p[2], n[2], 2, -p[0], -n[0]);
    j[2] = so * row(0, -p[1], -n[1], 1, p[0], n[0]);
#pragma unroll
    for (int c = 0; c < 3; c++)
        j[3 + c] = -weight * __fmaf_rn(-mz, T[8 + c], __fmaf_rn(-my, T[4 + c], -mx * T[c]));
}

// The arrays the photometric term reads: FP32, or (mixed precision) the FP16
// current image and reference intensities and the BF16 Jacobian.  Widening a
// stored FP16 / BF16 value to FP32 is exact, so the arithmetic that follows is
// the FP32 path's on rounded inputs.
template <bool kMixed> struct PhotoArrays;
template <> struct PhotoArrays<false> {
    using TI = float;
    using TJ = float;
    static __device__ const float *img(const InstDesc &d, int l) { return d.cur_gray[l]; }
    static __device__ const float *I(const InstDesc &d, int l) { return d.sel_I[l]; }
    static __device__ const float *J(const InstDesc &d, int l) { return d.sel_J[l]; }
};
template <> struct PhotoArrays<true> {
    using TI = __half;
    using TJ = __nv_bfloat16;
    static __device__ const __half *img(const InstDesc &d, int l) { return d.cur_grayh[l]; }
    static __device__ const __half *I(const InstDesc &d, int l) { return d.sel_Ih[l]; }
    static __device__ const __nv_bfloat16 *J(const InstDesc &d, int l) { return d.sel_Jb[l]; }
};

// Photometric residuals and depth weights of two points (interpolateResidualKernel2,
// warp.cu:269-332, the expressions of photo_residual) in the halves of register
// pairs: position p, keyframe intensity I.  Nothing branches on a point, so that
// the taps and the depth taps of all the points a thread evaluates are in flight
// together: the photometric term of a small batch is one chain of latencies.
// Points that fall outside read the image's first pixel and are set afterwards.
template <typename TImg>
__device__ __forceinline__ void photo_pair(const PhotoConsts &k, float2 one, const float2 *p, float2 I, const TImg *img,
                                           int w, int h, const float *zcur, int zw, int zh, float2 &res, float2 &zwt) {
    auto map = [&](const float2 *M, const float2 *v, float2 *o) {
#pragma unroll
        for (int i = 0; i < 3; i++)
            o[i] = plus2(add2(mul2(M[4 * i + 2], v[2]), add2(mul2(M[4 * i + 1], v[1]), mul2(M[4 * i], v[0]), one), one),
                         M[4 * i + 3]);
    };
    auto divide = [&](const float2 *v, float2 &x, float2 &y) {
        float2 nz = mul2(v[2], dup2(-1.0f)), r = rcp_rn2(v[2]);
        x = div_rn2(v[0], nz, r);
        y = div_rn2(v[1], nz, r);
        if (!div_in_range(v[0].x, v[1].x, v[2].x)) {
            x.x = ieee_div(v[0].x, v[2].x);
            y.x = ieee_div(v[1].x, v[2].x);
        }
        if (!div_in_range(v[0].y, v[1].y, v[2].y)) {
            x.y = ieee_div(v[0].y, v[2].y);
            y.y = ieee_div(v[1].y, v[2].y);
        }
    };
    // float -> int truncation of a coordinate, as an index >= 0 (the fraction
    // of a coordinate in (-1, 0) is itself: it truncates to 0)
    auto whole = [](float2 v) { return index_sum2(make_float2(fmaxf(v.x, 0.0f), fmaxf(v.y, 0.0f))); };
    float2 q[3], r[3], l[3], ux, uy, lx, ly;
    map(k.T, p, q);
    map(k.TLR, q, r);
    divide(r, ux, uy);
    // distortPoint
    float2 r2 = add2(mul2(uy, uy), mul2(ux, ux), one), r4 = mul2(r2, r2), r6 = mul2(r4, r2);
    float2 rad = add2(mul2(k.kc[2], r6), add2(mul2(k.kc[1], r4), add2(mul2(k.kc[0], r2), dup2(1.0f), one), one), one);
    float2 dx = add2(mul2(mul2(k.KR[0], ux), rad), k.KR[1], one), dy = add2(mul2(mul2(k.KR[2], uy), rad), k.KR[3], one);
    float2 px = add2(mul2(k.ab[0], dx), k.ab[1], one), py = add2(mul2(k.ab[0], dy), k.ab[1], one);
    float wm1 = (float)(w - 1), hm1 = (float)(h - 1);
    bool in0 = px.x > -1.0f && px.x < wm1 && py.x > -1.0f && py.x < hm1;
    bool in1 = px.y > -1.0f && px.y < wm1 && py.y > -1.0f && py.y < hm1;
    float2 sx = whole(px), sy = whole(py);
    const TImg *a = img + (in0 ? index_of(sx.x) + index_of(sy.x) * w : 0);
    const TImg *b = img + (in1 ? index_of(sx.y) + index_of(sy.y) * w : 0);
    float2 t0 = make_float2(ldf(a), ldf(b)), t1 = make_float2(ldf(a + 1), ldf(b + 1));
    float2 t2 = make_float2(ldf(a + w), ldf(b + w)), t3 = make_float2(ldf(a + w + 1), ldf(b + w + 1));
    // the depth at the nearest IR pixel
    map(k.TRL, r, l);
    divide(l, lx, ly);
    float2 vx = plus2(plus2(add2(mul2(k.KL[1], ly), mul2(k.KL[0], lx), one), k.KL[2]), dup2(0.5f));
    float2 vy = plus2(plus2(add2(mul2(k.KL[4], ly), mul2(k.KL[3], lx), one), k.KL[5]), dup2(0.5f));
    float zwf = (float)zw, zhf = (float)zh;
    bool zin0 = in0 && vx.x > -1.0f && vx.x < zwf && vy.x > -1.0f && vy.x < zhf;
    bool zin1 = in1 && vx.y > -1.0f && vx.y < zwf && vy.y > -1.0f && vy.y < zhf;
    float2 ix = whole(vx), iy = whole(vy);
    float2 zc = make_float2(__ldg(zcur + (zin0 ? index_of(ix.x) + index_of(iy.x) * zw : 0)),
                            __ldg(zcur + (zin1 ? index_of(ix.y) + index_of(iy.y) * zw : 0)));
    // bilinear tap and residual
    float2 u = sub2(px, whole_of2(sx)), v = sub2(py, whole_of2(sy));
    float2 gu = sub2(dup2(1.0f), u), gv = sub2(dup2(1.0f), v);
    float2 col = add2(mul2(mul2(u, v), t3),
                      add2(mul2(mul2(gu, v), t2), add2(mul2(mul2(u, gv), t1), mul2(mul2(gu, gv), t0), one), one), one);
    res = sub2(I, col);
    if (!in0) res.x = 1.0f;
    if (!in1) res.y = 1.0f;
    // 1 - (dz / 100)^2: the squared error over 1e4 by the exact division (below
    // its range the quotient leaves 1 as it is, however it is rounded)
    float2 e = sub2(zc, r[2]);
    e = mul2(e, e);
    float2 f = sub2(dup2(1.0f), div_rn2(e, dup2(-10000.0f), dup2(1.0f / 10000.0f)));
    zwt.x = zin0 && e.x < 10000.0f ? f.x : 0.0f;
    zwt.y = zin1 && e.y < 10000.0f ? f.y : 0.0f;
}

// The photometric term of an instance by its cluster of 8 CTAs: CTA `rank`
// evaluates chunks rank, rank + 8, ...; every CTA writes its histogram
// (histogram64.cu:115-145) into the others' shared memory, each finds the median
// bin (seekThreshold64Kernel, histogram64.cu:48-61) and weighs its own points
// (generateWeights64Kernel, 79-94) into the CTA's fixed-point sums.  In two
// parts: `photo_begin` before the kernels ahead have finished (constants, and
// the first chunk's points and Jacobian, which belong to the keyframe), the rest
// after.
struct PhotoLane {
    float2 p[2][3], I[2];  // the lane's points t + 256 m of the first chunk, m and m + 1 a pair
};

template <bool kMixed>
__device__ __forceinline__ void photo_load(const InstDesc &d, int level, int c, PhotoLane &o) {
    const auto *I = PhotoArrays<kMixed>::I(d, level);
#pragma unroll
    for (int g = 0; g < 2; g++) {
        int i = c * kChunk + threadIdx.x + 2 * g * kLanes;
#pragma unroll
        for (int k = 0; k < 3; k++)
            o.p[g][k] = make_float2(__ldg(d.sel_xyz + k * d.P + i), __ldg(d.sel_xyz + k * d.P + i + kLanes));
        o.I[g] = make_float2(ldf(I + i), ldf(I + i + kLanes));
    }
}

// the Jacobian tile in shared memory, in its stored type: column k of point i
// of the chunk at 1024 k + i (in 4-byte steps of 32 points, so that a warp's
// points are the runs of its reduction for either type)
template <typename TJ> __device__ __forceinline__ TJ *photo_tile(IterShared &sh, int col, int i) {
    return reinterpret_cast<TJ *>(&sh.stage[col * kChunk + (i & ~31)]) + (i & 31);
}

template <bool kMixed>
__device__ __forceinline__ void photo_begin(const InstDesc &d, IterShared &sh, int level, int rank, PhotoLane &o) {
    using TJ = typename PhotoArrays<kMixed>::TJ;
    int P = d.P, t = threadIdx.x;
    cluster_arrive();  // awaited before the first write to another CTA's shared memory
    if (rank < P / kChunk) {
        photo_load<kMixed>(d, level, rank, o);
        const TJ *J = PhotoArrays<kMixed>::J(d, level);
        constexpr int kPer16 = 16 / sizeof(TJ);  // values per 16-byte copy
        for (int k = t; k < 6 * (kChunk / kPer16); k += blockDim.x) {
            int col = k / (kChunk / kPer16), q = kPer16 * (k % (kChunk / kPer16));
            const TJ *src = J + (size_t)col * P + rank * kChunk + q;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                             (unsigned)__cvta_generic_to_shared(photo_tile<TJ>(sh, col, q))),
                         "l"(src)
                         : "memory");
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    sh.photo.set_level(d, level);
    for (int k = t; k < d.hist_bins; k += blockDim.x) sh.hist[k] = 0;
}

// Returns whether this CTA had a chunk.
template <bool kMixed>
__device__ bool photo_cluster(const InstDesc &d, IterShared &sh, int level, int rank, PhotoLane &lane0, uint32_t *sums,
                              int &bad) {
    using TJ = typename PhotoArrays<kMixed>::TJ;
    int P = d.P, nph = P / kChunk, nb = d.hist_bins;
    int t = threadIdx.x, lane = t & 31;
    int w = d.W >> level, h = d.H >> level;
    const auto *img = PhotoArrays<kMixed>::img(d, level);
    const float2 one = unseen_one();
    float2 r0[2], zw0[2];
    for (int c = rank; c < nph; c += kCluster) {
        if (c != rank) photo_load<kMixed>(d, level, c, lane0);
        float2 r[2], zw[2];
#pragma unroll
        for (int g = 0; g < 2; g++)
            photo_pair(sh.photo, one, lane0.p[g], lane0.I[g], img, w, h, d.cur_z, d.W, d.H, r[g], zw[g]);
#pragma unroll
        for (int g = 0; g < 2; g++) {
            atomicAdd(&sh.hist[mad_bin(r[g].x, nb)], 1);
            atomicAdd(&sh.hist[mad_bin(r[g].y, nb)], 1);
            if (c == rank) {
                r0[g] = r[g];
                zw0[g] = zw[g];
            } else {  // later chunks of this CTA go through global scratch
                int i = c * kChunk + t + 2 * g * kLanes;
                d.ph_r[i] = r[g].x;
                d.ph_r[i + kLanes] = r[g].y;
                d.ph_zw[i] = zw[g].x;
                d.ph_zw[i + kLanes] = zw[g].y;
            }
        }
    }
    __syncthreads();
    cluster_wait();  // every CTA of the cluster has begun
    for (int k = t; k < nb; k += blockDim.x) {
        int v = sh.hist[k];
#pragma unroll
        for (int q = 0; q < kCluster; q++) *cluster_peer(&sh.peers[rank][k], q) = v;
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    cluster_arrive();
    cluster_wait();  // every CTA's histogram is here (and no CTA touches another's memory from now on)
    // thread k: the instance's count of bin k; the median bin is the first
    // whose cumulative count exceeds P / 2
    int cnt = 0;
    if (t < nb) {
#pragma unroll
        for (int q = 0; q < kCluster; q++) cnt += sh.peers[q][t];
    }
    int incl = cnt;
    for (int o = 1; o < 32; o <<= 1) {
        int x = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += x;
    }
    if (lane == 31) sh.warp_tot[t >> 5] = incl;
    if (t == 0) sh.median = 0;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kIterThreads / 32; q++)
        if (q < (t >> 5)) incl += sh.warp_tot[q];
    if (t < nb && incl > P / 2 && incl - cnt <= P / 2) sh.median = t;
    __syncthreads();
    int median = sh.median;
    if (rank == 0) {
        if (t < nb) d.ph_hist[256 + t] = cnt;  // for the trace
        if (t == 0) d.ph_hist[512] = median;
    }
    // Tukey weights with the divisions by the scale and by the constant exact
    // (a quotient below the division's range leaves the weight as it is)
    float sc = mad_scale(median, nb), rsc = rcp_rn(sc);
    constexpr float kB = 4.6851f, kRb = 1.0f / 4.6851f;
    auto weight = [&](float2 r, float2 zw) {
        float2 u = div_rn2(make_float2(fabsf(r.x), fabsf(r.y)), dup2(-sc), dup2(rsc));
        float2 ub = div_rn2(u, dup2(-kB), dup2(kRb));
        float2 v = mul2(sub2(dup2(1.0f), mul2(ub, ub)), zw);
        return make_float2(u.x <= kB ? v.x : 0.0f, u.y <= kB ? v.y : 0.0f);
    };
    const TJ *J = PhotoArrays<kMixed>::J(d, level);
    for (int c = rank; c < nph; c += kCluster) {
        float acc[27];
#pragma unroll
        for (int q = 0; q < 27; q++) acc[q] = 0.0f;
#pragma unroll
        for (int g = 0; g < 2; g++) {
            int i = t + 2 * g * kLanes;
            float2 r, zw, j[6];
            if (c == rank) {
                r = r0[g];
                zw = zw0[g];
#pragma unroll
                for (int k = 0; k < 6; k++)
                    j[k] = make_float2((float)*photo_tile<TJ>(sh, k, i), (float)*photo_tile<TJ>(sh, k, i + kLanes));
            } else {
                int x = c * kChunk + i;  // written by this thread above
                r = make_float2(d.ph_r[x], d.ph_r[x + kLanes]);
                zw = make_float2(d.ph_zw[x], d.ph_zw[x + kLanes]);
#pragma unroll
                for (int k = 0; k < 6; k++) j[k] = make_float2(ldf(J + k * P + x), ldf(J + k * P + x + kLanes));
            }
            float2 wv = weight(r, zw);
            r = mul2(r, wv);
            float a[6];
#pragma unroll
            for (int k = 0; k < 6; k++) {
                j[k] = mul2(j[k], wv);
                a[k] = j[k].x;
            }
            acc27(acc, a, r.x);
#pragma unroll
            for (int k = 0; k < 6; k++) a[k] = j[k].y;
            acc27(acc, a, r.y);
        }
        fx_accumulate(sums, warp_terms(acc, sh.stage + (t & ~31)), bad);
    }
    return rank < nph;
}

// L2 prefetch of [p, p + bytes) (cp.async.bulk.prefetch.L2: a 16-byte aligned
// global address and a multiple of 16 bytes; a smaller tail is left out).  A
// prefetch changes no value anywhere, it only brings lines into L2 early.
__device__ __forceinline__ void prefetch_l2(const void *p, unsigned bytes) {
    bytes &= ~15u;
    if (bytes == 0) return;
    unsigned long long g;
    asm("cvta.to.global.u64 %0, %1;\n" : "=l"(g) : "l"(p));
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(g), "r"(bytes) : "memory");
}

// Prefetches what ICP chunk c of the level reads: its reference planes and
// weights (contiguous) and the rows of the current points that its taps read at
// small motion (the chunk's own rows and the one below).  Issued by one thread,
// a chunk ahead of its use.
__device__ __forceinline__ void icp_prefetch_chunk(const InstDesc &d, int level, int c, int npix) {
    int w = d.W >> level, h = d.H >> level, i0 = c * kChunk;
    if (i0 >= npix) return;
    prefetch_l2(d.ref_pl[level] + (size_t)c * 6 * kChunk, 6 * kChunk * 4);
    prefetch_l2(d.icp_w + i0, kChunk * 4);
    int y0 = i0 / w, y1 = min((min(i0 + kChunk, npix) - 1) / w + 1, h - 1);
    size_t first = (size_t)y0 * w, count = (size_t)(y1 - y0 + 1) * w;
    if (level == 0) {
        size_t down = first & 3;  // to a 16-byte boundary
        prefetch_l2(d.cur_z + first - down, (unsigned)(count + down) * 4u);
    } else {
        prefetch_l2(d.cur_pts[level] + first, (unsigned)count * 16u);
    }
}

// ICP chunks [c0, c1) of 1024 pixels of the level: lane t evaluates pixels
// t + 256m of each chunk, kBatch at a time with their inputs and then their taps
// in flight together, and leaves their terms in its own slots; the canonical
// per-lane sums then take them in pixel order, and the warp totals of each chunk
// go into the fixed-point sums that lane q keeps of term q.
template <bool kDepth>
__device__ void icp_chunks(const InstDesc &d, IterShared &sh, int level, int c0, int c1, int npix, uint32_t *sums,
                           int &bad) {
    // depths leave the registers for two pixels' taps at once (125 against 136 us
    // a level-0 launch of 30 instances), points do not (52 against 54 at level 1)
    constexpr int kBatch = kDepth ? 2 : 1;
    int t = threadIdx.x;
    const IcpLevel L(d, level);
    const float opt_in = d.opt_in;
    // a pixel's terms in the warp's own runs: three pairs, and the residual
    float *slot = sh.stage + ((t >> 4) & 1) * kChunk + (t & ~31) + 2 * (t & 15), *slot_r = sh.stage + 6 * kChunk + t;
    for (int c = c0; c < c1; c++) {
        if (t == 0 && c + 1 < c1) icp_prefetch_chunk(d, level, c + 1, npix);
        const float *ref = d.ref_pl[level] + (size_t)c * 6 * kChunk + t, *wts = d.icp_w + c * kChunk + t;
        // in registers: read from shared memory it would be read again after every
        // store to the slots (124 against 131 us at level 0 of 30 instances)
        float T[12];
#pragma unroll
        for (int k = 0; k < 12; k++) T[k] = sh.T[k];
#pragma unroll
        for (int g = 0; g < 4; g += kBatch) {
            IcpTaps<kDepth> tap[kBatch];
            float p[kBatch][6], w[kBatch], q[kBatch][3], px[kBatch], py[kBatch];
            bool in[kBatch];
#pragma unroll
            for (int u = 0; u < kBatch; u++) {
                w[u] = __ldcg(wts + (g + u) * kLanes);
#pragma unroll
                for (int k = 0; k < 6; k++) p[u][k] = __ldg(ref + k * kChunk + (g + u) * kLanes);
            }
#pragma unroll
            for (int u = 0; u < kBatch; u++) {
                mul4(T, p[u][0], p[u][1], p[u][2], q[u][0], q[u][1], q[u][2]);
                in[u] = w[u] > 0.0f && icp_project(L, q[u][0], q[u][1], q[u][2], px[u], py[u]);
                tap[u].load(L, icp_tap_index(L, in[u], px[u], py[u]));
            }
#pragma unroll
            for (int u = 0; u < kBatch; u++) {
                float j[6], r;
                icp_point<kDepth>(L, T, opt_in, w[u], p[u], p[u] + 3, q[u], px[u], py[u], in[u], tap[u], j, r);
                float *v = slot + (g + u) * kLanes;
#pragma unroll
                for (int k = 0; k < 3; k++)
                    *reinterpret_cast<float2 *>(v + 2 * k * kChunk) = make_float2(j[2 * k], j[2 * k + 1]);
                slot_r[(g + u) * kLanes] = r;
            }
        }
        Terms27 sum;
#pragma unroll
        for (int m = 0; m < 4; m++) {
            const float *v = slot + m * kLanes;
            sum.add(*reinterpret_cast<const float2 *>(v), *reinterpret_cast<const float2 *>(v + 2 * kChunk),
                    *reinterpret_cast<const float2 *>(v + 4 * kChunk), slot_r[m * kLanes]);
        }
        float acc[27];
        sum.terms(acc);
        fx_accumulate(sums, warp_terms(acc, sh.stage + (t & ~31)), bad);
    }
}

__device__ __forceinline__ int packed_index(int r, int c) {
    int a = r < c ? r : c, b = r < c ? c : r;
    return a * 6 - (a * (a - 1)) / 2 + (b - a);
}

// The end of an iteration of an instance: the accumulated terms in FP64, the
// system of the mode (fused in FP64 for BIOBJECTIVE with weights precomputed
// off this path, linearFuseKernel warp.cu:918-924), the solve and SE(3) update.
// Warp 0 takes the photometric terms (lane q: term q), warp 1 the ICP terms,
// handed over through shared memory; every global value is loaded in one round
// trip at the start, since the FP64 solve that follows is one serial chain on
// warp 0.  Warp 1 meanwhile resets the sums, keeps the work counters and writes
// the optional trace.  What bounds it is that chain, 64 cycles an FP64 instruction:
// about 7.5 of the 16.7 us of an iteration of 320x240 photometric tracking (one
// instance, graph replay), 3.4 us less than with the general exponential and a
// column-by-column Cholesky in place of solve.cuh's short forms.
__device__ __forceinline__ void finalize_iter(const InstDesc &d, SolveShared &sh, int level, int it, bool use_ph,
                                              bool use_icp) {
    int lane = threadIdx.x & 31, set = threadIdx.x >> 5;
    SolveScratch &S = sh.S;
    int q = lane < 27 ? lane : 26;
    unsigned long long *src = d.fx + set * kFxTerms + q * kFxLimbs;
    longlong2 l0 = __ldcg(reinterpret_cast<const longlong2 *>(src));
    longlong2 l1 = __ldcg(reinterpret_cast<const longlong2 *>(src) + 1);
    int bad = __ldcg(d.fx_bad + set);
    int nsel = use_icp ? __ldcg(d.icp_nsel + level) : 0;
    double c2 = __ldcg(d.fuse_c2 + level);
    int median = use_ph ? __ldcg(d.ph_hist + 512) : -1;
    float T_before = lane < 16 ? __ldcg(d.T + lane) : 0.0f;
    int st_iters = 0, st_solves = 0, st_nonspd = 0, slot = 0;
    unsigned long long work0 = 0, work1 = 0;
    if (set == 0) {
        st_iters = __ldcg(d.stats + ST_ITERS);
        st_solves = __ldcg(d.stats + ST_SOLVES);
        st_nonspd = __ldcg(d.stats + ST_NONSPD);
    } else {
        work0 = __ldcg(d.work + 0);
        work1 = __ldcg(d.work + 1);
    }
    if (d.trace) slot = __ldcg(d.trace_count);
    static_assert(kFxLimbs == 4, "two 16-byte loads per term");
    long long L[kFxLimbs] = {l0.x, l0.y, l1.x, l1.y};
    double term = bad ? __longlong_as_double(0x7ff8000000000000LL) : fx_to_double(L);
    if (set == 1) {
        if (lane < 27) sh.A_icp[lane] = term;
        if (lane < 16) S.T[lane] = (double)T_before;
    } else if (lane < 16) {
        sh.T[lane] = T_before;
    }
    bool ok = !(use_icp && nsel <= 0);  // ShapeTracker "not enough points": no solve
    recon_iter_trace *tr = d.trace && slot < d.trace_max ? d.trace + slot : nullptr;
    __syncthreads();
    // the packed term q of the mode's system
    auto fused = [&](double aph, double aic) {
        if (d.mode == RECON_PHOTOMETRIC) return aph;
        if (d.mode == RECON_GEOMETRIC) return aic;
        return ok ? __fma_rn(d.fuse_c1, aph, c2 * aic) : aph;  // (1-lambda)/P * photo + lambda/N * icp
    };
    if (set == 1) {
        ulonglong2 zero = make_ulonglong2(0ull, 0ull);
        for (int k = lane; k < 2 * kFxTerms / 2; k += 32) reinterpret_cast<ulonglong2 *>(d.fx)[k] = zero;
        if (lane < 2) d.fx_bad[lane] = 0;
        if (lane == 0) {
            if (use_ph) d.work[0] = work0 + (unsigned long long)d.P;
            if (use_icp) d.work[1] = work1 + (unsigned long long)nsel;
            if (use_icp) d.stats[ST_ICPSEL0 + level] = nsel;
            if (use_ph) d.stats[ST_MEDIAN] = median;
            if (d.trace) *d.trace_count = slot + 1;
        }
        if (tr) {
            for (int k = lane; k < 256; k += 32)
                tr->hist[k] = (use_ph && k < d.hist_bins) ? __ldcg(d.ph_hist + 256 + k) : 0;
            if (lane == 0) {
                tr->level = level;
                tr->iter = it;
                tr->mode = d.mode;
                tr->solved = ok ? 1 : 0;
                tr->icp_selected = use_icp ? nsel : 0;
                tr->median_bin = median;
            }
        }
        return;
    }
    double icp = sh.A_icp[q];
    double v = fused(term, icp);
    if (tr) {
        // the packed term's one or two entries of the full matrices
        for (int k = 0; k < 42; k++) {
            int qk = (k < 36) ? packed_index(k / 6, k % 6) : 21 + (k - 36);
            if (lane != qk) continue;
            if (k < 36) {
                tr->A[k] = v;
                tr->A_ph[k] = term;
                tr->A_icp[k] = icp;
            } else {
                tr->b[k - 36] = v;
                tr->b_ph[k - 36] = term;
                tr->b_icp[k - 36] = icp;
            }
        }
    }
    int st = 0;
    if (ok) st = wsolve_packed(S, d.solver, v, sh.T, (double)d.opt_out, lane);
    float T_after = lane < 16 ? sh.T[lane] : 0.0f;
    if (lane < 16) d.T[lane] = T_after;
    if (d.settle_mm > 0.0f) {
        // settle rule (orc_pose_settled): every translation entry moved by at
        // most settle_mm and every rotation entry by at most settle_rot; the
        // instance's remaining iterations of this level are skipped
        bool small = true;
        if (lane < 12) small = fabsf(T_after - T_before) <= ((lane & 3) == 3 ? d.settle_mm : d.settle_rot);
        if (__all_sync(0xffffffffu, small) && lane == 0) d.stats[ST_SETTLED] = level + 1;
    }
    if (tr && lane < 16) tr->T[lane] = T_after;
    if (lane == 0) {
        int *stt = d.stats;
        stt[ST_ITERS] = st_iters + 1;
        if (ok) stt[ST_SOLVES] = st_solves + 1;
        if (st != 0) stt[ST_NONSPD] = st_nonspd + 1;
        if (tr) tr->status = st;
    }
}


// The linearisation of one GN iteration at `level`, iteration `it`, for every
// instance.  The grid is one row: blocks [0, 8n) are the photometric clusters
// of the n instances (cluster i = instance i; updateLinearSystem,
// phototracker.cpp:505-511), then icp_ctas blocks per instance, block j of an
// instance taking ICP chunks [j K, (j+1) K) of 1024 pixels, K = icp_per_cta
// (ShapeTracker::updateLinearSystem, shapetracker.cpp:376-381).  The
// photometric clusters, the longest dependent chains of the iteration
// (residuals, a cluster-wide histogram, then the weighted sums), come first so
// that they all start in the first wave and the short ICP CTAs fill in around
// them.  Every CTA adds its fixed-point sums to the instance's with integer
// atomics, so the result does not depend on K or on the order in which CTAs
// finish; k_solve then fuses, solves and updates the pose.
//
// What bounds it: at the fine levels instruction issue, about 320 a pixel, and the
// latency of its taps (a level-0 launch of 30 640x480 instances moves 335 MB of
// DRAM, 49 us at the measured HBM rate, and takes 117 us; level 1 48 us), at the
// coarse levels and for a single instance the photometric chain (level 3 of 30
// instances 20 us; a 320x240 photometric iteration with its solve 16.7 us).
// Measured and not kept, on a scene whose level-0 launch takes 125 us: two pixels in
// packed arithmetic with the pose in shared memory (135 us: a third fewer
// instructions, but the constants' loads and 80 registers), inputs copied two
// blocks ahead into shared memory (3 CTAs an SM, of which clusters of 8 leave 11% of
// the slots empty: 134 us), one share of the blocks for each resident CTA (151 us:
// CTAs on SMs with fewer neighbours finish early).
//
// Even iterations visit the instances, and the chunks within each, in reverse
// order (CTAs start roughly in block order): a level-0 pass streams several
// times L2's capacity, and the lines it touched last (or k_icp_mask touched
// last, before iteration 0) are the ones the next pass then starts with.
#ifndef RECON_ITER_MIN_BLOCKS
#define RECON_ITER_MIN_BLOCKS 4
#endif
__global__ void __cluster_dims__(kCluster, 1, 1) __launch_bounds__(kIterThreads, RECON_ITER_MIN_BLOCKS)
    k_iter(const InstDesc *D, int level, int it, int icp_per_cta, int n_inst, int icp_ctas) {
    pdl_trigger();
    const bool rev = (it & 1) == 0;
    int slot, role;  // instance slot of the block, and its role within the instance
    if ((int)blockIdx.x < kCluster * n_inst) {
        slot = blockIdx.x / kCluster;
        role = blockIdx.x % kCluster;
    } else {
        int j = blockIdx.x - kCluster * n_inst;
        if (icp_ctas <= 0) return;
        slot = j / icp_ctas;
        role = kCluster + j % icp_ctas;
        if (slot >= n_inst) return;  // rounding of the grid to whole clusters
    }
    __shared__ InstDesc sd;
    __shared__ IterShared sh;
    load_desc(sd, D + (rev ? n_inst - 1 - slot : slot));
    __syncthreads();
    const InstDesc &d = sd;
    if (level >= d.L) return;
    if (it >= d.iters[d.L - 1 - level]) return;
    const bool icp = role >= kCluster;
    if (icp ? d.mode == RECON_PHOTOMETRIC : d.mode == RECON_GEOMETRIC) return;
    int npix = (d.W >> level) * (d.H >> level);
    int nchunks = (npix + kChunk - 1) / kChunk;
    int nicp = (nchunks + icp_per_cta - 1) / icp_per_cta;
    int j = role - kCluster;
    if (icp && j >= nicp) return;
    int c0 = (rev ? nicp - 1 - j : j) * icp_per_cta, c1 = min(c0 + icp_per_cta, nchunks);
    // what does not depend on the kernels before: the first chunk's inputs into
    // L2, or the photometric term's constants, points and Jacobian
    if (icp && threadIdx.x == 0) icp_prefetch_chunk(d, level, c0, npix);
    const bool mixed = d.precision == RECON_PRECISION_MIXED;
    PhotoLane first;
    if (!icp) {
        if (mixed) photo_begin<true>(d, sh, level, role, first);
        else photo_begin<false>(d, sh, level, role, first);
    }
    if (threadIdx.x == 0) sh.bad = 0;
    pdl_wait();
    float pose = threadIdx.x < 16 ? __ldcg(d.T + threadIdx.x) : 0.0f;
    // the instance left this level early (settle rule; uniform over a cluster),
    // or it has no correspondence there
    bool skip = d.settle_mm > 0.0f && __ldcg(d.stats + ST_SETTLED) == level + 1;
    if (icp && __ldcg(d.icp_nsel + level) <= 0) skip = true;
    if (threadIdx.x < 16) sh.T[threadIdx.x] = pose;
    if (!icp) sh.photo.set_pose(pose);
    __syncthreads();
    if (skip) {
        if (!icp) {
            cluster_wait();
            asm volatile("cp.async.wait_all;\n" ::: "memory");
        }
        return;
    }
    uint32_t sums[kFxLimbs] = {0u, 0u, 0u, 0u};
    int bad = 0;
    if (icp) {
        if (level == 0) icp_chunks<true>(d, sh, level, c0, c1, npix, sums, bad);
        else icp_chunks<false>(d, sh, level, c0, c1, npix, sums, bad);
    } else {
        bool had = mixed ? photo_cluster<true>(d, sh, level, role, first, sums, bad)
                         : photo_cluster<false>(d, sh, level, role, first, sums, bad);
        if (!had) return;
    }
    int set = icp ? 1 : 0;  // which sums this CTA adds to: 0 photometric, 1 ICP
    fx_flush(sh, sums, bad, d.fx + set * kFxTerms, d.fx_bad + set);
}

// The rest of a GN iteration, one CTA per instance after k_iter: the normal
// equations from the fixed-point sums, fusion, solve and SE(3) update
// (estimateIncrement, phototracker.cpp:646-664; linearFuse,
// shapetracker.cpp:392-394).
__global__ void __launch_bounds__(kSolveThreads) k_solve(const InstDesc *D, int level, int it) {
    pdl_trigger();
    __shared__ InstDesc sd;
    load_desc(sd, D + blockIdx.x);
    __syncthreads();
    const InstDesc &d = sd;
    if (level >= d.L) return;
    if (it >= d.iters[d.L - 1 - level]) return;
    pdl_wait();
    if (d.settle_mm > 0.0f && __ldcg(d.stats + ST_SETTLED) == level + 1) return;
    bool use_ph = d.mode != RECON_GEOMETRIC;
    bool use_icp = d.mode != RECON_PHOTOMETRIC;
    __shared__ SolveShared sh;
    finalize_iter(d, sh, level, it, use_ph, use_icp);
}

// The whole ICP preparation of a small level in one launch: the level's
// correspondences (k_icp_mask's per-pixel work), their count and first
// variance sum, and the three Student-t passes (updateWeightsKernel /
// clampWeightsKernel, rgb2gray.cu:549-569): each pass weighs every
// correspondence with the variance of the previous pass; the final pass
// clamps at 1 and writes every pixel's weight (0 where the pixel is not a
// correspondence), the first two produce only their variance sums (exact int64
// sums of truncated products).  An 8-CTA cluster per instance (blockIdx.y)
// splits the pixels, every thread reading back only what it wrote, and
// exchanges the CTAs' sums through distributed shared memory, so no pass waits
// for a separate launch.  Two CTAs fit on an SM, so a batch of up to 38
// instances runs in one wave.
constexpr int kStudentThreads = 1024;

__device__ __forceinline__ void student_body(const InstDesc *D, int level) {
    __shared__ InstDesc sd;
    __shared__ float sT[16];
    __shared__ long long part[3];
    __shared__ int part_cnt;
    __shared__ long long warp_sum[kStudentThreads / 32];
    __shared__ int warp_cnt[kStudentThreads / 32];
    __shared__ long long s_var0;
    __shared__ int s_nsel;
    load_desc(sd, D + blockIdx.y);
    __syncthreads();
    const InstDesc &d = sd;
    if (level >= d.L || d.mode == RECON_PHOTOMETRIC) return;
    if (d.iters[d.L - 1 - level] <= 0) return;  // uniform over the cluster
    pdl_wait();
    int n = (d.W >> level) * (d.H >> level);
    int rank = blockIdx.x, t = threadIdx.x, lane = t & 31, wid = t >> 5;
    int stride = kIterCluster * kStudentThreads;
    int c = 0;
    long long v = 0;
    {
        if (t < 16) sT[t] = __ldcg(d.T + t);
        if (rank == 0 && t == 0) d.work[2] += (unsigned long long)n;
        __syncthreads();
        const IcpLevel L(d, level);
        const StudentW first(100.0f);
        const float *pl = d.ref_pl[level];
        for (int i0 = rank * kStudentThreads + t; i0 < n; i0 += 2 * stride) {
            // two pixels at a time: point and normal loads in flight together
            float p[2][6];
#pragma unroll
            for (int u = 0; u < 2; u++)
#pragma unroll
                for (int k = 0; k < 6; k++)
                    p[u][k] = i0 + u * stride < n ? __ldg(pl + ref_plane(i0 + u * stride, k)) : 0.0f;
#pragma unroll
            for (int u = 0; u < 2; u++) {
                int i = i0 + u * stride;
                if (i >= n) continue;
                float r2;
                bool ok = level == 0 ? icp_mask_pixel<true>(L, sT, p[u], r2) : icp_mask_pixel<false>(L, sT, p[u], r2);
                if (ok) v += trunc_prod(r2, first(r2));
                d.icp_r2[i] = r2;
                d.icp_mask[i] = ok;
                c += ok;
            }
        }
    }
    c = __reduce_add_sync(0xffffffffu, c);
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) {
        warp_cnt[wid] = c;
        warp_sum[wid] = v;
    }
    __syncthreads();
    if (t == 0) {
        int cs = 0;
        long long vs = 0;
        for (int w = 0; w < kStudentThreads / 32; w++) {
            cs += warp_cnt[w];
            vs += warp_sum[w];
        }
        part[2] = vs;
        part_cnt = cs;
    }
    cluster_arrive();
    cluster_wait();  // every CTA's count and first sum are in its shared memory
    if (t == 0) {
        int cs = 0;
        long long vs = 0;
#pragma unroll
        for (int r = 0; r < kIterCluster; r++) {
            cs += *cluster_peer(&part_cnt, r);
            vs += *cluster_peer(&part[2], r);
        }
        s_nsel = cs;
        s_var0 = vs;
    }
    __syncthreads();
    int nsel = s_nsel;
    long long var = s_var0;
    if (rank == 0 && t == 0) {
        d.icp_nsel[level] = nsel;
        // ICP weight of the fused system, kept off the iteration's critical path
        d.fuse_c2[level] = (double)d.lambda / (double)nsel;
        d.icp_var[0] = (unsigned long long)var;
    }
    for (int pass = 1; pass <= 3; pass++) {
        float Sf = (float)var;
        float minVal = (float)nsel;
        float vv = (nsel <= 1024) ? Sf : (Sf < minVal ? minVal : Sf);
        const StudentW weight(vv / (float)nsel);
        long long vsum = 0;
        int i = rank * kStudentThreads + t;
        float r_next = 0.0f;
        uint8_t m_next = 0;
        if (i < n) {
            r_next = d.icp_r2[i];
            m_next = d.icp_mask[i];
        }
        for (; i < n; i += stride) {
            // the next pixel's loads are in flight while this one is weighed
            float r = r_next;
            uint8_t mk = m_next;
            if (i + stride < n) {
                r_next = d.icp_r2[i + stride];
                m_next = d.icp_mask[i + stride];
            }
            if (pass == 3) {
                d.icp_w[i] = mk ? fminf(weight(r), 1.0f) : 0.0f;
            } else if (mk) {
                vsum += trunc_prod(r, weight(r));
            }
        }
        if (pass == 3) {
            // zero up to the end of the level's last block
            for (int k = n + rank * kStudentThreads + t; k < (n + kChunk - 1) / kChunk * kChunk; k += stride) d.icp_w[k] = 0.0f;
            break;
        }
        for (int o = 16; o > 0; o >>= 1) vsum += __shfl_xor_sync(0xffffffffu, vsum, o);
        if (lane == 0) warp_sum[wid] = vsum;
        __syncthreads();
        if (t == 0) {
            long long sum = 0;
            for (int w = 0; w < kStudentThreads / 32; w++) sum += warp_sum[w];
            part[pass - 1] = sum;
        }
        cluster_arrive();
        cluster_wait();  // every CTA's sum of this pass is in its shared memory
        long long tot = 0;
#pragma unroll
        for (int r = 0; r < kIterCluster; r++) tot += *cluster_peer(&part[pass - 1], r);
        var = tot;
        if (rank == 0 && t == 0) d.icp_var[pass] = (unsigned long long)tot;
        __syncthreads();  // warp_sum is rewritten by the next pass
    }
    // no CTA leaves while another may still read its sums
    cluster_arrive();
    cluster_wait();
}

// The coarser levels' ICP preparation, where the grid is small enough for one
// cluster per instance to evaluate it.  Two CTAs per SM (a few registers spill
// in the mask phase; measured faster than one CTA per SM at 30 instances).
__global__ void __cluster_dims__(kIterCluster, 1, 1) __launch_bounds__(kStudentThreads, 2)
    k_icp_prepare(const InstDesc *D, int level) {
    pdl_trigger();
    student_body(D, level);
}

// ------------------------------------------------------------------
// learned initialisation: network inputs and the start-pose gate
// ------------------------------------------------------------------

// Coarse network image ([60][80][2] BF16: gray, depth in metres / 4) of each
// instance's uint8 / uint16 input frame, from the input pointer table
// (gray pointers, then depth pointers); the formula of recon_initnet_coarse.
__global__ void __launch_bounds__(256) k_net_coarse(const InstDesc *D, const uint8_t *const *in_gray,
                                                     const uint16_t *const *in_depth, const __nv_bfloat16 *prev,
                                                     __nv_bfloat16 *out, __nv_bfloat16 *net_in) {
    const InstDesc &d = D[blockIdx.y];
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= kNetW * kNetH) return;
    const uint8_t *g = in_gray[blockIdx.y];
    const uint16_t *dp = in_depth[blockIdx.y];
    if (!g || !dp) return;
    int W = d.W, bx = d.W / kNetW, by = d.H / kNetH;
    int ox = p % kNetW, oy = p / kNetW;
    int gs = 0, cnt = 0;
    long long ds = 0;
    for (int y = 0; y < by; y++)
        for (int x = 0; x < bx; x++) {
            long long o = (long long)(oy * by + y) * W + ox * bx + x;
            gs += __ldg(g + o);
            int dv = __ldg(dp + o);
            if (dv) {
                ds += dv;
                cnt++;
            }
        }
    float gv = (float)gs / (255.0f * (float)(bx * by));
    float dv = cnt ? ((float)ds / (float)cnt) / 4000.0f : 0.0f;
    long long q = (long long)blockIdx.y * kNetW * kNetH + p;
    __nv_bfloat16 bg = __float2bfloat16_rn(gv), bd = __float2bfloat16_rn(dv);
    out[2 * q] = bg;
    out[2 * q + 1] = bd;
    if (net_in) {  // the network input (previous gray, depth, current gray, depth)
        net_in[4 * q + 0] = prev[2 * q];
        net_in[4 * q + 1] = prev[2 * q + 1];
        net_in[4 * q + 2] = bg;
        net_in[4 * q + 3] = bd;
    }
}

// Integer start-pose cost of one point: min(trunc(|r| * 1024), 1024) of its
// photometric residual at `level`.
__device__ __forceinline__ long long gate_cost_point(const InstDesc &d, const float *T, int level, int i) {
    int P = d.P, w = d.W >> level, h = d.H >> level;
    float a = 1.0f / (float)(1 << level);
    float b = 0.5f * (a - 1.0f);
    float r, zw;
    photo_residual(d.calib, T, a, b, __ldg(d.sel_xyz + i), __ldg(d.sel_xyz + P + i), __ldg(d.sel_xyz + 2 * P + i),
                   __ldg(d.sel_I[level] + i), d.cur_gray[level], w, h, d.cur_z, d.W, d.H, r, zw);
    float u = fabsf(r) * 1024.0f;
    return (u >= 1024.0f || !(u == u)) ? 1024 : (long long)(int)u;  // 0 <= u < 1024: a 32-bit conversion
}

// The learned start pose, step 1 (one warp per instance, no pose needed, so it
// runs with the network): the network's twist x = out * scale (FP32) mapped to
// D = exp(A(x)) applied to the identity (wexpm_update, FP64, the tracker's own
// pose update), stored as the float matrix the candidate D * T is formed from.
__global__ void __launch_bounds__(32) k_gate_twist(const InstDesc *D, const float *net_out, const float *scale,
                                                   float *Dout) {
    const InstDesc &d = D[blockIdx.x];
    __shared__ float Dm[16];
    __shared__ SolveScratch S;
    int t = threadIdx.x;
    if (t < 16) {
        Dm[t] = (t % 5 == 0) ? 1.0f : 0.0f;
        S.T[t] = (t % 5 == 0) ? 1.0 : 0.0;
    }
    __syncwarp();
    double x[6];
    for (int k = 0; k < 6; k++) x[k] = (double)(net_out[blockIdx.x * 6 + k] * scale[k]);
    wexpm_update(S, x, Dm, (double)d.opt_out, t);
    if (t < 16) Dout[16 * blockIdx.x + t] = Dm[t];
}

// Step 2 (grid: point blocks x instances): the candidate Tc = D * T from the
// previous pose T (FP32, as the oracle forms it), the integer costs of T and of
// Tc at the coarsest level (exact integer sums, any order), and in the
// instance's last CTA to finish (an atomic ticket) the choice: Tc replaces T
// when its cost is strictly lower.  That CTA resets the costs and the ticket
// for the next frame.
__global__ void __launch_bounds__(256) k_gate(const InstDesc *D, const float *Dm_all, long long *cost,
                                              unsigned int *ticket, float *cand, int *choice) {
    __shared__ InstDesc sd;
    __shared__ float Tp[16], Tc[16];
    __shared__ long long part[2][8];
    __shared__ bool last;
    load_desc(sd, D + blockIdx.y);
    __syncthreads();
    const InstDesc &d = sd;
    int t = threadIdx.x, inst = blockIdx.y;
    if (t < 16) Tp[t] = __ldcg(d.T + t);
    __syncthreads();
    if (t < 16) {
        const float *Dm = Dm_all + 16 * inst;
        int r = t >> 2, c = t & 3;
        Tc[t] = Dm[r * 4 + 0] * Tp[0 * 4 + c] + Dm[r * 4 + 1] * Tp[1 * 4 + c] + Dm[r * 4 + 2] * Tp[2 * 4 + c] +
                Dm[r * 4 + 3] * Tp[3 * 4 + c];
    }
    __syncthreads();
    int level = d.L - 1;
    long long c0 = 0, c1 = 0;
    for (int i = blockIdx.x * blockDim.x + t; i < d.P; i += gridDim.x * blockDim.x) {
        c0 += gate_cost_point(d, Tp, level, i);
        c1 += gate_cost_point(d, Tc, level, i);
    }
    for (int o = 16; o > 0; o >>= 1) {
        c0 += __shfl_xor_sync(0xffffffffu, c0, o);
        c1 += __shfl_xor_sync(0xffffffffu, c1, o);
    }
    if ((t & 31) == 0) {
        part[0][t >> 5] = c0;
        part[1][t >> 5] = c1;
    }
    __syncthreads();
    if (t == 0) {
        long long s0 = 0, s1 = 0;
        for (int w = 0; w < 8; w++) {
            s0 += part[0][w];
            s1 += part[1][w];
        }
        atomicAdd(reinterpret_cast<unsigned long long *>(cost + 2 * inst), (unsigned long long)s0);
        atomicAdd(reinterpret_cast<unsigned long long *>(cost + 2 * inst + 1), (unsigned long long)s1);
        __threadfence();
        last = atomicAdd(ticket + inst, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    // every CTA's costs are in: the choice
    __threadfence();
    long long k0 = (long long)__ldcg(reinterpret_cast<unsigned long long *>(cost + 2 * inst));
    long long k1 = (long long)__ldcg(reinterpret_cast<unsigned long long *>(cost + 2 * inst + 1));
    bool take = k1 < k0;
    if (t < 16) {
        cand[16 * inst + t] = Tc[t];
        if (take) d.T[t] = Tc[t];
    }
    if (t == 0) {
        if (choice) choice[inst] = take ? 1 : 0;
        cost[2 * inst] = 0;
        cost[2 * inst + 1] = 0;
        ticket[inst] = 0u;
    }
}

// ------------------------------------------------------------------
// procedural renderer
// ------------------------------------------------------------------

__global__ void k_render_depth(recon_scene sc, recon_camera cam, float noise_rel, uint32_t seed, uint32_t frame,
                               uint16_t *out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cam.width * cam.height) return;
    out[i] = scene_depth_pixel(&sc, &cam, i % cam.width, i / cam.width, noise_rel, seed, frame);
}

__global__ void k_render_gray(recon_scene sc, recon_camera cam, uint8_t *out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cam.width * cam.height) return;
    out[i] = scene_gray_pixel(&sc, &cam, i % cam.width, i / cam.width);
}

}  // namespace rt

// ====================================================================
// Allocation-free photometric iteration.
//
// Some callers cannot allocate device memory while they track: a host that
// runs the tracker inside a real-time frame loop, where a cudaMalloc can
// synchronise the device and stall the frame, or a host framework that owns
// all device memory through its own allocator and hands plug-ins only the
// buffers it created.  For them this variant of the photometric GN iteration
// keeps its scratch (per-point residuals and depth weights) in a file-scope
// device array instead of per-instance buffers from cudaMalloc.
//
// The array is a static __device__ symbol: every GPU that loads the library
// holds it until the process exits, and every call shares it and finds the
// previous call's contents there.  Calls that overlap on the GPU (different
// streams, or different host threads on the same device) race on it and must
// be serialised by the caller.  Nothing in it has to start at zero: the
// residual and weight slots for the call's points are written before they
// are read, and the partial sums live in shared memory.
// ====================================================================

namespace rt {

constexpr int kNoAllocMaxPoints = RECON_NOALLOC_MAX_POINTS;

// residual[P], depth weight[P]: 128 KB for the 16384-point maximum
static __device__ __align__(256) float g_noalloc_scratch[2 * kNoAllocMaxPoints];

__global__ void __launch_bounds__(256) k_photo_iter_noalloc(recon_photo_view v, float *scratch, float *T) {
    __shared__ PhotoShared sh;
    __shared__ InstDesc d;  // view of the caller's buffers in the layout photo_iteration reads
    if (threadIdx.x == 0) {
        d.W = v.depth_width;
        d.H = v.depth_height;
        d.P = v.n_points;
        d.hist_bins = v.hist_bins;
        for (int i = 0; i < RECON_CALIB_SIZE; i++) d.calib[i] = v.calib[i];
        for (int l = 0; l < kMaxLevels; l++) {
            d.cur_gray[l] = nullptr;
            d.sel_I[l] = nullptr;
            d.sel_J[l] = nullptr;
        }
        d.cur_gray[v.level] = const_cast<float *>(v.img);
        d.sel_I[v.level] = const_cast<float *>(v.intensity);
        d.sel_J[v.level] = const_cast<float *>(v.jacobian);
        d.sel_xyz = const_cast<float *>(v.xyz);
        d.cur_z = const_cast<float *>(v.depth);
        d.ph_r = scratch;
        d.ph_zw = scratch + kNoAllocMaxPoints;
    }
    if (threadIdx.x < 16) sh.T[threadIdx.x] = T[threadIdx.x];
    __syncthreads();
    photo_iteration(d, sh, v.level);
    __syncthreads();
    if (threadIdx.x >= 32) return;
    int lane = threadIdx.x;
    SolveScratch &S = sh.S;
    for (int k = lane; k < 42; k += 32) {
        int q = (k < 36) ? packed_index(k / 6, k % 6) : 21 + (k - 36);
        if (k < 36) S.A[k] = sh.A_ph[q];
        else S.b[k - 36] = sh.A_ph[q];
    }
    __syncwarp();
    wsolve_update(S, v.solver, sh.T, (double)v.opt_scale_out, lane);
    if (lane < 16) T[lane] = sh.T[lane];
}

}  // namespace rt

namespace rt {
void set_last_error(const char *msg);
}

namespace {
std::mutex g_noalloc_mu;
void *g_noalloc_ptr[64] = {nullptr};

int noalloc_reject(const char *msg) {
    rt::set_last_error(msg);
    return RECON_ERR_INVALID_ARG;
}
}  // namespace

extern "C" int recon_photometric_iteration_noalloc(const recon_photo_view *v, float *T_dev, void *stream) {
    if (!v || !T_dev || !v->xyz || !v->intensity || !v->jacobian || !v->img || !v->depth)
        return noalloc_reject("recon_photometric_iteration_noalloc: null pointer");
    if (v->n_points <= 0 || v->n_points % rt::kChunk)
        return noalloc_reject("recon_photometric_iteration_noalloc: n_points must be a positive multiple of 1024");
    if (v->n_points > rt::kNoAllocMaxPoints)
        return noalloc_reject("recon_photometric_iteration_noalloc: n_points exceeds RECON_NOALLOC_MAX_POINTS "
                              "(16384), the size of the built-in scratch array");
    if (v->level < 0 || v->level >= rt::kMaxLevels || v->hist_bins < 2 || v->hist_bins > 256)
        return noalloc_reject("recon_photometric_iteration_noalloc: level must be 0..3 and hist_bins 2..256");
    if (v->img_width < 2 || v->img_height < 2 || v->img_width != (v->depth_width >> v->level) ||
        v->img_height != (v->depth_height >> v->level))
        return noalloc_reject("recon_photometric_iteration_noalloc: img must be the depth size >> level");
    if (v->solver < 0 || v->solver > 1) return noalloc_reject("recon_photometric_iteration_noalloc: bad solver");
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        rt::set_last_error("recon_photometric_iteration_noalloc: no current CUDA device");
        return RECON_ERR_CUDA;
    }
    void *ptr = nullptr;
    {
        // set-up, once per device with that device current: the host-side name
        // of a __device__ array is not a device address, so look it up
        std::lock_guard<std::mutex> lk(g_noalloc_mu);
        if (!g_noalloc_ptr[dev]) {
            cudaError_t e = cudaGetSymbolAddress(&g_noalloc_ptr[dev], rt::g_noalloc_scratch);
            if (e != cudaSuccess) {
                g_noalloc_ptr[dev] = nullptr;
                rt::set_last_error("recon_photometric_iteration_noalloc: cudaGetSymbolAddress failed");
                return RECON_ERR_CUDA;
            }
        }
        ptr = g_noalloc_ptr[dev];
    }
    // the launch status comes from the launch call itself, so an error the
    // caller's own earlier work left pending is neither cleared nor taken for ours
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1);
    cfg.blockDim = dim3(rt::kLanes);
    cfg.stream = (cudaStream_t)stream;
    cudaError_t e = cudaLaunchKernelEx(&cfg, rt::k_photo_iter_noalloc, *v, (float *)ptr, T_dev);
    if (e != cudaSuccess) {
        rt::set_last_error("recon_photometric_iteration_noalloc: kernel launch failed");
        return RECON_ERR_CUDA;
    }
    return RECON_OK;
}
