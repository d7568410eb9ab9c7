// tsdf.cu -- the reconstruction stream: TSDF fusion of distance maps into a
// voxel grid, ray casting and shading of the fused surface, resampling of a
// grid into a moved frame, and the distance map of an RGB-D frame.
//
// Reference: tracker/kernels/VoxelGrid_cuda.cu (kernels) and
// tracker/reconstruct/VoxelGrid.cpp (host object).  Every per-voxel and
// per-pixel value is the reference's arithmetic in its source order (the
// library is built with -fmad=false; divisions and square roots are IEEE);
// float -> unsigned conversions saturate as the reference's make_uint3 and
// `uint += float` do on the GPU.  What differs is how the work is mapped:
//
//  * update: a CTA takes a 32x8x8 block of voxels, each thread a run of 8 voxels
//    along z at one (x, y), so that a warp reads and writes 32 consecutive
//    float2 (256 bytes).  A block whose voxel centres all project outside the
//    image (tested at its 8 corners, with a margin for rounding) is skipped
//    as a whole: the projection is a linear-fractional map, so over a box on
//    one side of the camera plane its extremes lie at the corners.  On large
//    grids a block that lies behind all distances its pixels show is skipped
//    too, and the blocks to visit are listed first.  A voxel is written only
//    when its value changes.
//  * ray cast: one thread per pixel, one warp per 8x4 tile.  A byte per 8x8x8 brick
//    records whether any voxel of the brick may be negative; the traversal
//    steps through bricks without one using only its step arithmetic (the
//    reference's coarse test, tsdf < 0, cannot pass there), so empty space
//    costs no grid reads, and many such bricks are crossed at one go.  The byte is set whenever a negative value is
//    stored and cleared only by a reset or a rebuild, so it never hides a
//    negative voxel.
//  * where the reference would read past the end of the grid array (its
//    bounds checks are commented out), a ray reports no hit.
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <utility>
#include <vector>

#include "../../include/recon_track.h"
#include "../../include/recon_tsdf.h"
#include "pair_math.cuh"

namespace rt {
void set_last_error(const char *msg);
void add_launches(long long n);
}  // namespace rt

namespace tsdf {

constexpr int kBrick = 8;    // voxels per side of a flag brick
constexpr int kTileX = 32;   // update CTA: 32 x 8 columns of 8 voxels along z
constexpr int kTileY = 8;
constexpr int kRunZ = 8;
constexpr int kFarTile = 16;    // distance map tiles of the update's test for blocks behind the surface
constexpr int kFarMost = 256;   // tiles that a block may look at
constexpr int kUpdateCtas = 8;  // CTAs per SM of an update: 32 registers
// From this many blocks on the update picks the blocks to visit first: two small
// launches more, which have to save more than they cost on a single grid.  The
// update of one grid by itself, 640x480 frames of a room, all blocks / picked ones:
// 192^3 (3456 blocks) 29 / 38 us, 256^3 (8192) 51 / 59, 320^3 (16000) 90 / 99, 352^3
// (21296) 117 / 116, 512^3 (65536) 344 / 339.  (What picking saves depends on how
// much of the grid lies behind surfaces.  With the frames of three grids on their
// streams, where other work fills the launches' gaps, four scenes on 256^3 took
// 762, 805, 753 and 766 us with all blocks, 745, 818, 746 and 751 with picked ones.)
constexpr int kListBlocks = 18000;
constexpr int kRayTileX = 8;  // ray cast CTA: one warp on 8 x 4 pixels (rays differ widely in length;
constexpr int kRayTileY = 4;  // one-warp CTAs let the block scheduler balance the SMs)
constexpr int kRayCtas = 28;  // ray cast CTAs per SM: 72 registers.  32 (64 registers) spill more and 24 leave fewer
                              // rays to switch between: 796, 779 and 791 us for six 640x480 frames on a 256^3 grid
constexpr int kKinds = 5;     // timing kinds: update, ray cast, shading, distance map, reset / resample

struct Geom {
    int R, B, SB, W, H;             // voxels, 8^3 bricks and 32^3 super bricks per side, image size
    int tiles_x, tiles_y;           // 16 x 16 tiles of the distance map
    int nb;                         // B^3: offset of the super-brick bytes
    float T[12];                    // update: world -> camera; ray cast / resample: camera -> world
    float K0, K2, K4, K5, Wf, Hf, Wm2, Hm2;
    float sx, sy, sz;               // centre of voxel 0 (start)
    float vx2, vy2, vz2;            // voxel spacing (2 * voxelSize)
    float lim, tol, slope, inv_slope, slope_lo;  // update gates; RN(1 / slope), the least numerator for div_rn
    float b0x, b0y, b0z, b1x, b1y, b1z;  // grid bounds
    float ib0x, ib0y, ib0z;         // interpolation origin
    float ivx, ivy, ivz;            // 1 / voxel spacing (voxelize's invVoxelDim)
    float min_dist, max_dist;
    int mirror;      // 2^k - 1 >= R - 1
    int exact_walk;  // every corner coordinate of a voxel walk is an exact sum
};

__device__ __forceinline__ unsigned f2u(float v) { return __float2uint_rz(v); }

__device__ __forceinline__ size_t brick_of(const Geom &g, unsigned x, unsigned y, unsigned z) {
    return ((size_t)(z >> 3) * g.B + (y >> 3)) * g.B + (x >> 3);
}
__device__ __forceinline__ size_t super_of(const Geom &g, unsigned x, unsigned y, unsigned z) {
    return (size_t)g.nb + ((size_t)(z >> 5) * g.SB + (y >> 5)) * g.SB + (x >> 5);
}
// marks the brick and super brick of a voxel that holds a negative value
__device__ __forceinline__ void mark_negative(uint8_t *flags, const Geom &g, unsigned x, unsigned y, unsigned z) {
    flags[brick_of(g, x, y, z)] = 1;
    flags[super_of(g, x, y, z)] = 1;
}

// ---------------------------------------------------------------- update --

// programmatic dependent launches (launch_after)
__device__ __forceinline__ void wait_before() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void next_may_start() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

// The largest distance in each 16 x 16 tile of the distance map (infinity where
// the tile holds a NaN): one warp per tile.
__global__ void __launch_bounds__(128) k_far_tiles(const float *__restrict__ dist, Geom g, float *__restrict__ far_tiles,
                                                   int *__restrict__ counts) {
    next_may_start();
    if (blockIdx.x == 0 && threadIdx.x < 2) counts[threadIdx.x] = 0;
    const int tile = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (tile >= g.tiles_x * g.tiles_y) return;
    const int x = (tile % g.tiles_x) * kFarTile + (lane & 15), y0 = (tile / g.tiles_x) * kFarTile + (lane >> 4);
    float far = 0.0f;
#pragma unroll
    for (int k = 0; k < kFarTile; k += 2) {
        const float d = x < g.W && y0 + k < g.H ? __ldg(dist + (size_t)(y0 + k) * g.W + x) : 0.0f;
        far = d == d ? fmaxf(far, d) : __int_as_float(0x7f800000);
    }
    for (int o = 16; o; o >>= 1) far = fmaxf(far, __shfl_xor_sync(0xffffffffu, far, o));
    if (lane == 0) far_tiles[tile] = far;
}

// The 32 x 8 x 8 block of voxels at (x0, y0, z0), by its corner voxel centres:
// one per lane of a group of 8 lanes (all 32 lanes take part).
struct Block {
    float lo_x, hi_x, lo_y, hi_y;  // pixels
    float near;                    // the least depth, less what the roundings may add
    bool outside;                  // no voxel projects into the image
    bool sharp;                    // in front of the camera, projected to better than a pixel
    bool plain;                    // in front of it, and no coordinate beyond the range of div_rn
    __device__ __forceinline__ Block(const Geom &g, int x0, int y0, int z0) {
        const int lane = threadIdx.x & 31, group = lane & 24;
        const int cx = min(x0 + ((lane & 1) ? kTileX - 1 : 0), g.R - 1);
        const int cy = y0 + ((lane & 2) ? kTileY - 1 : 0), cz = z0 + ((lane & 4) ? kRunZ - 1 : 0);
        const float px = g.sx + (float)cx * g.vx2, py = g.sy + (float)cy * g.vy2, pz = g.sz + (float)cz * g.vz2;
        const float rx = g.T[0] * px + g.T[1] * py + g.T[2] * pz + g.T[3];
        const float ry = g.T[4] * px + g.T[5] * py + g.T[6] * pz + g.T[7];
        const float rz = g.T[8] * px + g.T[9] * py + g.T[10] * pz + g.T[11];
        lo_x = hi_x = (rx / rz * g.K0 + g.K2) * g.Wf;
        lo_y = hi_y = (ry / rz * g.K4 + g.K5) * g.Hf;
        const float off = 1e-6f * (fabsf(g.T[8] * px) + fabsf(g.T[9] * py) + fabsf(g.T[10] * pz) + fabsf(g.T[11]));
        near = -rz - off;
        const bool small = fmaxf(fmaxf(fabsf(rx), fabsf(ry)), -rz) <= 0x1p40f;
        const bool pixel = off * fmaxf(fabsf(g.K0) * g.Wf, fabsf(g.K4) * g.Hf) < near;
        for (int o = 1; o < 8; o <<= 1) {
            lo_x = fminf(lo_x, __shfl_xor_sync(0xffffffffu, lo_x, o));
            hi_x = fmaxf(hi_x, __shfl_xor_sync(0xffffffffu, hi_x, o));
            lo_y = fminf(lo_y, __shfl_xor_sync(0xffffffffu, lo_y, o));
            hi_y = fmaxf(hi_y, __shfl_xor_sync(0xffffffffu, hi_y, o));
            near = fminf(near, __shfl_xor_sync(0xffffffffu, near, o));
        }
        // |rz| >= 16 mm at every corner keeps the rounding of the projected
        // coordinates far below the 4-pixel margin
        // (votes of all lanes: none may depend on another's outcome)
        const unsigned front = __ballot_sync(0xffffffffu, rz < -16.0f) >> group & 0xffu;
        const unsigned behind = __ballot_sync(0xffffffffu, rz > 16.0f) >> group & 0xffu;
        const unsigned to_pixel = __ballot_sync(0xffffffffu, pixel) >> group & 0xffu;
        const unsigned all_small = __ballot_sync(0xffffffffu, small) >> group & 0xffu;
        sharp = front == 0xffu && to_pixel == 0xffu;
        plain = front == 0xffu && all_small == 0xffu && fmaxf(fabsf(g.K0), fabsf(g.K4)) <= 16.0f;
        outside = (front == 0xffu || behind == 0xffu) && (!(hi_x >= -3.0f) || !(lo_x < g.Wf + 2.0f) ||
                                                          !(hi_y >= -3.0f) || !(lo_y < g.Hf + 2.0f));
    }
    // Whether the block lies behind all that its pixels show: every distance
    // that its voxels can see is too short for them to be fused.  A slack of 4
    // pixels and of 1e-4 covers the roundings of the projection, of the
    // interpolated distance and of the quotient.
    // (far_tiles is written while the kernel that reads it already waits: a plain
    // load, not one for read-only memory.)
    __device__ __forceinline__ bool hidden(const Geom &g, const float *far_tiles) const {
        const int lane = threadIdx.x & 31;
        const int tx0 = (int)fmaxf(lo_x - 4.0f, 0.0f) / kFarTile, ty0 = (int)fmaxf(lo_y - 4.0f, 0.0f) / kFarTile;
        const int tx1 = (int)fminf(hi_x + 6.0f, g.Wf - 1.0f) / kFarTile;
        const int ty1 = (int)fminf(hi_y + 6.0f, g.Hf - 1.0f) / kFarTile;
        const int nx = tx1 - tx0 + 1, n = nx * (ty1 - ty0 + 1);
        const bool look = sharp && !outside && n <= kFarMost;
        float far = 0.0f;
        if (look)
            for (int i = lane & 7; i < n; i += 8) far = fmaxf(far, far_tiles[(ty0 + i / nx) * g.tiles_x + tx0 + i % nx]);
        for (int o = 1; o < 8; o <<= 1) far = fmaxf(far, __shfl_xor_sync(0xffffffffu, far, o));
        return look && (far < g.lim || near - far > 1.25f * g.slope + 1e-4f * (near + g.slope));
    }
};

// The blocks that the update has to visit: 8 lanes per block.  count was set
// to 0 by k_far_tiles.  A block that is not plain is listed as ~number.  Their
// order in the list is of no matter: every voxel is in one block.
__global__ void __launch_bounds__(256)
    k_pick_blocks(const float *far_tiles, Geom g, int bx, int by, int n, int *list, int *count) {
    next_may_start();
    const int lane = threadIdx.x & 31, i = (blockIdx.x * 256 + threadIdx.x) >> 3, b = min(i, n - 1);
    const Block block(g, b % bx * kTileX, b / bx % by * kTileY, b / bx / by * kRunZ);
    wait_before();
    const bool hidden = block.hidden(g, far_tiles);  // by all lanes
    const bool visit = (lane & 7) == 0 && i < n && !hidden && !block.outside;
    const unsigned all = __ballot_sync(0xffffffffu, visit);
    int at = 0;
    if (lane == 0 && all) at = atomicAdd(count, __popc(all));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (visit) list[at + __popc(all & ((1u << lane) - 1))] = block.plain ? b : ~b;
}

// updateVoxelsKernel (VoxelGrid_cuda.cu:944-1014) for the 8 voxels along z from
// (ix, iy, z0)
//
// plain (Block::plain, uniform over the warp): the quotients of the projection go
// through div_rn without a look at the operands.  They are at most 2^40; one below
// 2^-60, or a zero whose sign is lost, moves the pixel by less than 2^-60 of the
// image: nothing beside a principal point of 2^-20, and with a smaller one the
// pixel is before the first.
__device__ __forceinline__ void fuse_run(float2 *__restrict__ grid, uint8_t *__restrict__ flags,
                                         const float *__restrict__ dist, const Geom &g, bool plain, int ix, int iy,
                                         int z0, unsigned &n_proj, unsigned &n_fused, unsigned &n_changed) {
    const float px = g.sx + (float)ix * g.vx2;
    const float py = g.sy + (float)iy * g.vy2;
    // T p summed left to right: the first two products do not depend on z
    const float ax = g.T[0] * px + g.T[1] * py, ay = g.T[4] * px + g.T[5] * py, az = g.T[8] * px + g.T[9] * py;
    const size_t slice = (size_t)g.R * g.R;
    float2 *gp = grid + (size_t)z0 * slice + (size_t)iy * g.R + ix;
    float zf = (float)z0;
    // the run lies in one brick
    uint8_t *brick = flags + brick_of(g, ix, iy, z0), *super = flags + super_of(g, ix, iy, z0);
#pragma unroll 2
    for (int k = 0; k < kRunZ; k++, gp += slice, zf += 1.0f) {
        const float pz = g.sz + zf * g.vz2;
        const float rx = ax + g.T[2] * pz + g.T[3];
        const float ry = ay + g.T[6] * pz + g.T[7];
        const float rz = az + g.T[10] * pz + g.T[11];
        const float voxel_dist = -rz;
        const float irz = rt::rcp_rn(rz);
        float qx = rt::div_rn(rx, voxel_dist, irz), qy = rt::div_rn(ry, voxel_dist, irz);
        if (!plain) {
            qx = rt::ieee_div(rx, rz);
            qy = rt::ieee_div(ry, rz);
        }
        const float ux = (qx * g.K0 + g.K2) * g.Wf;
        const float uy = (qy * g.K4 + g.K5) * g.Hf;
        // int(u) in [1, size - 2): the reference's safeBorder of 1
        if (!(ux >= 1.0f && ux < g.Wm2 && uy >= 1.0f && uy < g.Hm2)) continue;
        n_proj++;
        // trunc by a sum rounded toward zero: no conversions
        const float su = rt::index_sum(ux), sv = rt::index_sum(uy);
        const float *dp = dist + (rt::index_of(sv) * g.W + rt::index_of(su));
        const float a = __ldg(dp), b = __ldg(dp + 1), c = __ldg(dp + g.W), d = __ldg(dp + g.W + 1);
        if (fminf(fminf(a, b), fminf(c, d)) < g.lim) continue;
        const float fu = ux - (su - 8388608.0f);
        const float fv = uy - (sv - 8388608.0f);
        const float z = (1 - fu) * (1 - fv) * a + fu * (1 - fv) * b + (1 - fu) * fv * c + fu * fv * d;
        if (fabsf(z - a) > g.tol || fabsf(z - b) > g.tol || fabsf(z - c) > g.tol || fabsf(z - d) > g.tol) continue;
        const float dz = -(voxel_dist - z);
        float sdf = rt::div_rn(dz, -g.slope, g.inv_slope);
        if (!(fabsf(dz) >= g.slope_lo && fabsf(dz) <= 0x1p60f)) sdf = rt::ieee_div(dz, g.slope);
        if (sdf < -1.25f) continue;
        n_fused++;
        const float nt = fmaxf(fminf(1.0f, sdf), -1.0f);
        const float2 old = *gp;
        const float nx = (old.y * old.x + nt) / (old.y + 1.0f);
        const float ny = fminf(1.0f + old.y, 16.0f);
        if (__float_as_uint(nx) != __float_as_uint(old.x) || __float_as_uint(ny) != __float_as_uint(old.y)) {
            *gp = make_float2(nx, ny);
            n_changed++;
        }
        if (nx < 0.0f) *brick = *super = 1;
    }
}

// All blocks of the grid.  counts (kCount): voxels [projected into the image,
// fused, changed].  As many CTAs per SM as the listed update has, for the latency
// of its gathers: 256^3 51 us, 512^3 344; 53 and 373 at the registers it would take.
template <bool kCount>
__global__ void __launch_bounds__(kTileX * kTileY, kUpdateCtas)
    k_update(float2 *__restrict__ grid, uint8_t *__restrict__ flags, const float *__restrict__ dist, Geom g,
             unsigned long long *__restrict__ counts) {
    __shared__ int s_skip;
    const int lane = threadIdx.x & 31;
    const int x0 = blockIdx.x * kTileX, y0 = blockIdx.y * kTileY, z0 = blockIdx.z * kRunZ;
    if (threadIdx.x < 32) {
        const Block block(g, x0, y0, z0);
        if (lane == 0) s_skip = block.outside ? 1 : (block.plain ? 0 : 2);
    }
    __syncthreads();
    if (s_skip == 1) return;
    const int ix = x0 + lane, iy = y0 + (threadIdx.x >> 5);
    if (ix >= g.R) return;
    unsigned n_proj = 0, n_fused = 0, n_changed = 0;
    fuse_run(grid, flags, dist, g, s_skip == 0, ix, iy, z0, n_proj, n_fused, n_changed);
    if (kCount) {
        n_proj = __reduce_add_sync(0xffffffffu, n_proj);
        n_fused = __reduce_add_sync(0xffffffffu, n_fused);
        n_changed = __reduce_add_sync(0xffffffffu, n_changed);
        if (lane == 0) {
            atomicAdd(&counts[0], (unsigned long long)n_proj);
            atomicAdd(&counts[1], (unsigned long long)n_fused);
            atomicAdd(&counts[2], (unsigned long long)n_changed);
        }
    }
}

// The blocks of k_pick_blocks' list, each taken by the next CTA that is free
// (counts: the blocks listed, and those taken).  What bounds it is instruction
// issue, about 110 a voxel and 63% of the slots.  On a 512^3 grid, of whose voxels
// a frame has 57% outside the image and 18 to 32% hidden behind the surface, all
// three launches of the listed update take 280 us; 346 with the blocks dealt out
// evenly beforehand (kListBlocks has a CTA for each block of the grid beside it).
// More voxels in flight per thread (2, 4 or 8 along z loaded together) were slower.
__global__ void __launch_bounds__(kTileX * kTileY, kUpdateCtas)
    k_update_list(float2 *__restrict__ grid, uint8_t *__restrict__ flags, const float *__restrict__ dist, Geom g, int bx,
                  int by, const int *list, int *counts) {
    wait_before();
    __shared__ int s_next[2];
    const int n = counts[0], lane = threadIdx.x & 31, row = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_next[0] = atomicAdd(counts + 1, 1);
    __syncthreads();
    for (int turn = 0; s_next[turn] < n; turn ^= 1) {
        const int entry = list[s_next[turn]], b = entry < 0 ? ~entry : entry;
        // the next one is asked for while this one is worked on
        int next = 0;
        if (threadIdx.x == 0) next = atomicAdd(counts + 1, 1);
        const int ix = b % bx * kTileX + lane;
        unsigned n_proj = 0, n_fused = 0, n_changed = 0;
        if (ix < g.R)
            fuse_run(grid, flags, dist, g, entry >= 0, ix, b / bx % by * kTileY + row, b / bx / by * kRunZ, n_proj, n_fused,
                     n_changed);
        if (threadIdx.x == 0) s_next[turn ^ 1] = next;
        __syncthreads();
    }
}

// -------------------------------------------------------------- ray cast --

// trilinearDensity / trilinearWeight (VoxelGrid_cuda.cu:181-260) at q (voxel
// units), channel ch; false when a corner lies past the end of the array
__device__ __forceinline__ bool trilinear(const float2 *__restrict__ grid, const Geom &g, float qx, float qy,
                                          float qz, int ch, float *out) {
    const unsigned ix = f2u(qx), iy = f2u(qy), iz = f2u(qz);
    const float fx = qx - (float)ix, fy = qy - (float)iy, fz = qz - (float)iz;
    const size_t ys = (size_t)g.R, zs = ys * g.R;
    const size_t o = (size_t)ix + (size_t)iy * ys + (size_t)iz * zs;
    if (o + 1 + ys + zs >= zs * g.R) return false;
    const float *f = reinterpret_cast<const float *>(grid) + ch;
    const float d000 = __ldg(f + 2 * o);
    const float d001 = __ldg(f + 2 * (o + zs));
    const float d010 = __ldg(f + 2 * (o + ys));
    const float d011 = __ldg(f + 2 * (o + ys + zs));
    const float d100 = __ldg(f + 2 * (o + 1));
    const float d101 = __ldg(f + 2 * (o + 1 + zs));
    const float d110 = __ldg(f + 2 * (o + 1 + ys));
    const float d111 = __ldg(f + 2 * (o + 1 + ys + zs));
    const float x00 = (1 - fx) * d000 + fx * d100;
    const float x01 = (1 - fx) * d001 + fx * d101;
    const float x10 = (1 - fx) * d010 + fx * d110;
    const float x11 = (1 - fx) * d011 + fx * d111;
    const float z0 = (1 - fy) * x00 + fy * x10;
    const float z1 = (1 - fy) * x01 + fy * x11;
    *out = (1 - fz) * z0 + fz * z1;
    return true;
}

// estimateLinearZero (VoxelGrid_cuda.cu:553-557)
__device__ __forceinline__ float linear_zero(float tA, float dA, float tB, float dB) {
    const float s = fmaxf(0.0f, fminf(dA / (dA - dB), 1.0f));
    return tA + s * (tB - tA);
}

struct Ray {
    float ox, oy, oz, dx, dy, dz;
};

__device__ __forceinline__ bool sample(const float2 *__restrict__ grid, const Geom &g, const Ray &r, float ivx,
                                       float ivy, float ivz, float t, float *out) {
    return trilinear(grid, g, (r.ox + t * r.dx - g.ib0x) * ivx, (r.oy + t * r.dy - g.ib0y) * ivy,
                     (r.oz + t * r.dz - g.ib0z) * ivz, 0, out);
}

// 2: the voxel's 32^3 super brick holds no negative value; 1: its 8^3 brick
// holds none; 0: the voxel may be negative, or lies outside [0, R)^3 (where
// the reference's flattened index wraps into the next row or slice)
__device__ __forceinline__ int empty_level(const uint8_t *__restrict__ flags, const Geom &g, int x, int y, int z) {
    const unsigned R = (unsigned)g.R;
    if (!((unsigned)x < R && (unsigned)y < R && (unsigned)z < R)) return 0;
    // both bytes are asked for at once: the second is no slower than the first
    const uint8_t sup = __ldg(flags + super_of(g, x, y, z)), brick = __ldg(flags + brick_of(g, x, y, z));
    return sup == 0 ? 2 : (brick == 0 ? 1 : 0);
}

// traverseVoxelsCuda's fine search once the coarse test passed
// (VoxelGrid_cuda.cu:674-704): 1 hit, 0 no hit (the traversal ends), 2 the
// trilinear value at the voxel is not negative (the traversal goes on)
__device__ __forceinline__ int refine(const float2 *__restrict__ grid, const Geom &g, const Ray &r, float ivx,
                                      float ivy, float ivz, float vpx, float vpy, float vpz, float enterT,
                                      float exitT, int iter, int max_back, unsigned rays, float *t_hit) {
    const float dv = (vpx - r.ox) * r.dx + (vpy - r.oy) * r.dy + (vpz - r.oz) * r.dz;
    float t1 = fmaxf(enterT, fminf(dv, exitT));
    float e1;
    int result = 0;
    if (sample(grid, g, r, ivx, ivy, ivz, t1, &e1)) result = e1 < 0.0f ? 1 : 2;
    // back in half-voxel steps to a positive value: a loop of its own, so that
    // the rays of a warp go into the bisection together
    float t0 = t1 - g.vx2 / 2, e0 = 0.0f;
    bool found = false;
    for (int back = 0; result == 1 && t0 > enterT && back < max_back; back++) {
        if (!sample(grid, g, r, ivx, ivy, ivz, t0, &e0)) break;
        found = e0 > 0.0f;
        if (found) break;
        if (e0 > e1) {
            t1 = t0;
            e1 = e0;
        }
        t0 -= g.vx2 * 0.5f;
    }
    if (result == 1 && !found) result = 0;
    __syncwarp(rays);
    if (result != 1) return result;
    float tx = linear_zero(t0, e0, t1, e1);
    for (; iter > 0; iter--) {
        float ex;
        if (!sample(grid, g, r, ivx, ivy, ivz, tx, &ex)) return 0;
        if (ex < 0.0f) {
            t1 = tx;
            e1 = ex;
        } else {
            t0 = tx;
            e0 = ex;
        }
        tx = linear_zero(t0, e0, t1, e1);
    }
    *t_hit = tx;
    return 1;
}

// Repeated addition T += ts without taking every step.  While T stays in one
// binade [2^e, 2^(e+1)) each sum is a multiple of the binade's unit u, so every
// addition rounds ts to the same multiple d of u and k of them give T + k d,
// one exact multiply-add.  Where ts lies half-way between two multiples the
// sum is rounded to an even one: from an even T that is again the same d, from
// an odd T only once (`even` is then false and one addition is taken).
struct Binade {
    float d, top;
    bool even;
    __device__ __forceinline__ Binade(float T, float ts) {
        const unsigned b = __float_as_uint(T), e = b & 0x7f800000u;
        top = __uint_as_float(e + 0x00800000u);
        d = (T + ts) - T;
        const float half = __uint_as_float(e - (24u << 23));
        // T in [2^-101, 2^126], positive
        even = b - (26u << 23) < 0x7e000000u - (26u << 23) && d > 0.0f && !((b & 1u) && fabsf(ts - d) == half);
    }
    // T after k additions; at least top where not all of them stay below it
    __device__ __forceinline__ float after(float T, int k) const { return __fmaf_rn((float)k, d, T); }
};

// One axis of the voxel walk: the next plane-crossing time, its step and the
// step's reciprocal (an estimate); the voxel index, its direction, and the
// events taken.
struct Moment {
    float tn, ts, rts;
};
struct Axis : Moment {
    int c, d, n;
    __device__ __forceinline__ void step(bool yes) {
        if (yes) tn += ts;
        took(yes);
    }
    __device__ __forceinline__ void took(int k) {
        c = max(c + d * k, 0);
        n += k;
    }
    // the events before the one that leaves the S-block (S = 8 or 32, the
    // block also ending at R); -1 when none leaves it (the index saturates at 0
    // in block 0)
    __device__ __forceinline__ int to_boundary(int S, int R) const {
        return d > 0 ? min(S - 1 - (c & (S - 1)), R - 1 - c) : (c >= S ? (c & (S - 1)) : -1);
    }
};

// the time of the event after `left` more events
__device__ __forceinline__ float time_after(Moment A, int left) {
    while (left > 0) {
        const Binade B(A.tn, A.ts);
        const int k = min(left, max((int)((B.top - A.tn) * A.rts), 0));
        const float t = B.after(A.tn, k);
        if (B.even && t < B.top) {
            A.tn = t;
            left -= k;
        }
        if (left > 0) {
            A.tn += A.ts;
            left--;
        }
    }
    return A.tn;
}

// takes the events before time Te (those at Te too with `at`); how many, or
// more than `most` where there are more than that
__device__ __forceinline__ int pass(Moment &A, float Te, bool at, int most) {
    int n = 0;
    while ((A.tn < Te || (at && A.tn == Te)) && n <= most) {
        const Binade B(A.tn, A.ts);
        int k = min(max((int)((fminf(Te, B.top) - A.tn) * A.rts), 0), most);
        float t = B.after(A.tn, k);
        if (!(t < Te)) t = B.after(A.tn, --k);
        if (B.even && t < B.top && t < Te && k > 0) {
            A.tn = t;
            n += k;
        }
        A.tn += A.ts;
        n++;
    }
    return n;
}

// A voxel corner's coordinate after n steps, carried along when the fine
// search asks for it.  exact: every such sum is exact (walk_is_exact), so the
// steps are one multiply-add.
struct Corner {
    float vp, gs;
    int n;
    __device__ __forceinline__ float at(int k, bool exact) {
        if (exact)
            vp = __fmaf_rn((float)(k - n), gs, vp);
        else
            for (int i = n; i < k; i++) vp += gs;
        n = k;
        return vp;
    }
};

// traverseVoxelsCuda (VoxelGrid_cuda.cu:628-730).  The voxel coordinates are
// kept as ints: the reference steps them with `uint += float` by +-1, which
// for coordinates below 2^24 is an integer step that saturates at 0.
//
// The reference's walk is a merge of three per-axis event sequences (plane
// crossings at tn, tn + ts, ...; each value depends only on how many steps its
// own axis took): at every step it takes the axis with the smallest tn, ties
// going to z, then y, then x.  So the order of all events is the order of
// (time, z < y < x).  Where the walk is after an event therefore depends on
// that event alone, not on how it got there, and while the voxels that it
// passes hold no negative value nothing else of it matters.  So empty blocks
// (32^3 super bricks and 8^3 bricks without a negative value) are crossed in
// two parts: block after block by times estimated with one rounding, for as
// long as the estimates' error bound leaves no doubt about the block that the
// walk is in, and then to the event that enters the block where that ends,
// exactly: its time, the other axes' events before it, and their times are
// those of the reference's additions (time_after, pass).  Where two boundaries
// are too close to call, the first of them is found by its exact time.  Voxels
// that may hold a negative value, and those outside [0, R)^3, are visited one
// by one, as the reference does.
//
// What bounds it is instruction issue (58% of the slots; DRAM 2%), so the rays
// of a warp are kept on the same part of the walk: all cross empty blocks, then
// all walk, and the fine search waits until none can walk on.  640x480 rays on
// a 256^3 grid of a room take 57.4 million warp instructions and 148 us; 95.6
// million and 193 us with every block crossed axis by axis in loops of additions.
__device__ bool traverse(bool in_grid, const float2 *__restrict__ grid, const uint8_t *__restrict__ flags, const Geom &g,
                         const Ray &r, float idx, float idy, float idz, int s0, int s1, int s2, float enterT,
                         float exitT, int iter, float *t_hit) {
    const float vdx = g.vx2, vdy = g.vy2, vdz = g.vz2;
    enterT += vdx * 2;
    exitT -= vdx * 2;
    if (enterT < 0) enterT = 0;
    if (enterT + vdx * 2 > exitT) in_grid = false;
    const float ivx = g.ivx, ivy = g.ivy, ivz = g.ivz;
    const unsigned vx = f2u((r.ox + enterT * r.dx - g.ib0x) * ivx);
    const unsigned vy = f2u((r.oy + enterT * r.dy - g.ib0y) * ivy);
    const unsigned vz = f2u((r.oz + enterT * r.dz - g.ib0z) * ivz);
    // the start point lies in the grid box, so its voxel is in [0, R]^3
    if (vx > (unsigned)g.R + 1 || vy > (unsigned)g.R + 1 || vz > (unsigned)g.R + 1) in_grid = false;
    const float sgx = (float)(1 - 2 * s0), sgy = (float)(1 - 2 * s1), sgz = (float)(1 - 2 * s2);
    Corner px = {g.ib0x + (float)vx * vdx, sgx * vdx, 0};
    Corner py = {g.ib0y + (float)vy * vdy, sgy * vdy, 0};
    Corner pz = {g.ib0z + (float)vz * vdz, sgz * vdz, 0};
    Axis X, Y, Z;
    X.tn = (px.vp + px.gs - r.ox) * idx;
    Y.tn = (py.vp + py.gs - r.oy) * idy;
    Z.tn = (pz.vp + pz.gs - r.oz) * idz;
    X.ts = px.gs * idx;
    Y.ts = py.gs * idy;
    Z.ts = pz.gs * idz;
    X.rts = rt::rcp_approx(X.ts);
    Y.rts = rt::rcp_approx(Y.ts);
    Z.rts = rt::rcp_approx(Z.ts);
    X.d = 1 - 2 * s0;
    Y.d = 1 - 2 * s1;
    Z.d = 1 - 2 * s2;
    X.c = (int)vx;
    Y.c = (int)vy;
    Z.c = (int)vz;
    X.n = Y.n = Z.n = 0;
    const size_t R = (size_t)g.R, RR = R * R, nvox = RR * R;
    const float *gx = reinterpret_cast<const float *>(grid);
    // a ray crosses at most R + 2 voxel planes per axis inside the grid and
    // the fine search steps back at most 4R + 4 half voxels; the caps end the
    // loops only where float steps stall (a grid far from the origin with tiny
    // voxels), where the reference's loops would not end
    const int max_steps = 3 * g.R + 16, max_back = 4 * g.R + 16;
    int at_x = 0, at_y = 0, at_z = 0;
    // voxels counted along the walk: w = c ^ m ascends on every axis, and 8 and
    // 32 blocks stay blocks; the last one that the walk may leave on each axis
    const int mx = s0 ? g.mirror : 0, my = s1 ? g.mirror : 0, mz = s2 ? g.mirror : 0;
    // a bound on the distance of an estimated event time from its sum: R + 3
    // roundings of at most 2^-24 of the largest, taken twice over.  It needs
    // times of the ray's own size; a ray along a grid axis has others.
    float err = (float)(g.R + 4) * 1.1920929e-7f * exitT;
    const float voxel_err = (float)g.R * 5e-7f;  // of a position in voxels, by the reciprocal and the roundings
    {
        const auto plain = [&](const Axis &A) { return A.tn >= -exitT && A.tn < 1e30f && A.ts > 1e-30f && A.ts < 1e30f; };
        if (!(plain(X) && plain(Y) && plain(Z))) err = __int_as_float(0x7f800000);
    }
    int steps = 0;
    float t = enterT;
    enum { kWalk, kFine, kMiss, kHit };
    int state = in_grid && t < exitT ? kWalk : kMiss;
    int lvl = state == kWalk ? empty_level(flags, g, X.c, Y.c, Z.c) : 0;
    while (true) {
        // the fine search waits until no ray of the warp can walk on
        if (!__any_sync(0xffffffffu, state == kWalk)) {
            const unsigned rays = __ballot_sync(0xffffffffu, state == kFine);
            if (!rays) break;
            if (state == kFine) {
                const int rr = refine(grid, g, r, ivx, ivy, ivz, px.at(at_x, g.exact_walk), py.at(at_y, g.exact_walk),
                                      pz.at(at_z, g.exact_walk), enterT, exitT, iter, max_back, rays, t_hit);
                state = rr == 1 ? kHit : (rr == 2 && t < exitT ? kWalk : kMiss);
            }
            continue;
        }
        // blocks without a negative value, by estimated times
        bool fast = state == kWalk && lvl > 0;
        bool stuck = false;
        int ea = -1, left = 0;
        float Te = 0.0f;
        if (fast) {
            const int cx = X.c ^ mx, cy = Y.c ^ my, cz = Z.c ^ mz;
            const int lim_x = (g.R - 1) | mx, lim_y = (g.R - 1) | my, lim_z = (g.R - 1) | mz;
            int wx = cx, wy = cy, wz = cz;
            int S = lvl == 2 ? 32 : 8;
            while (true) {
                // the last voxel of the block on each axis, and the time of the event that leaves it
                const int ux = min(wx | (S - 1), lim_x), uy = min(wy | (S - 1), lim_y), uz = min(wz | (S - 1), lim_z);
                const float Ex = __fmaf_rn((float)(ux - cx), X.ts, X.tn), Ey = __fmaf_rn((float)(uy - cy), Y.ts, Y.tn),
                            Ez = __fmaf_rn((float)(uz - cz), Z.ts, Z.tn);
                const float E = fminf(fminf(Ex, Ey), Ez);
                const float second = fmaxf(fminf(Ex, Ey), fminf(fmaxf(Ex, Ey), Ez));
                if (E > exitT + err) {
                    state = kMiss;
                    break;
                }
                const bool isx = E == Ex, isy = E == Ey;
                const int u = isx ? ux : (isy ? uy : uz), base = isx ? cx : (isy ? cy : cz);
                if (!(E + 2.0f * err < fminf(second, exitT)) || u == (isx ? lim_x : (isy ? lim_y : lim_z))) break;
                ea = isx ? 0 : (isy ? 1 : 2);
                left = u - base;
                // the other axes' voxels at that time, if all estimates within
                // the error agree on the brick
                const float qx = fmaxf(__fmaf_rn(E - X.tn, X.rts, (float)(cx + 1)), (float)cx),
                            qy = fmaxf(__fmaf_rn(E - Y.tn, Y.rts, (float)(cy + 1)), (float)cy),
                            qz = fmaxf(__fmaf_rn(E - Z.tn, Z.rts, (float)(cz + 1)), (float)cz);
                const float dx = __fmaf_rn(err, X.rts, voxel_err), dy = __fmaf_rn(err, Y.rts, voxel_err),
                            dz = __fmaf_rn(err, Z.rts, voxel_err);
                wx = isx ? u + 1 : rt::index_of(rt::index_sum(qx + dx));
                wy = !isx && isy ? u + 1 : rt::index_of(rt::index_sum(qy + dy));
                wz = !isx && !isy ? u + 1 : rt::index_of(rt::index_sum(qz + dz));
                int apart = 0;
                if (!isx) apart |= wx ^ rt::index_of(rt::index_sum(fmaxf(qx - dx, 0.0f)));
                if (isx || !isy) apart |= wy ^ rt::index_of(rt::index_sum(fmaxf(qy - dy, 0.0f)));
                if (isx || isy) apart |= wz ^ rt::index_of(rt::index_sum(fmaxf(qz - dz, 0.0f)));
                if (apart >> 3) break;
                if (max(wx - lim_x, max(wy - lim_y, wz - lim_z)) > 0) break;
                const int vx_ = wx ^ mx, vy_ = wy ^ my, vz_ = wz ^ mz;
                const int ib = ((vz_ >> 3) * g.B + (vy_ >> 3)) * g.B + (vx_ >> 3);
                const int is = ((vz_ >> 5) * g.SB + (vy_ >> 5)) * g.SB + (vx_ >> 5);
                const uint8_t sup = __ldg(flags + g.nb + is), brick = __ldg(flags + ib);
                S = sup == 0 ? 32 : 8;
                if (sup != 0 && brick != 0) break;
            }
        }
        __syncwarp();
        fast = fast && state == kWalk;
        if (fast) {
            // the event that leaves the last of them, or the first in (time,
            // z < y < x) order of those that may leave the first
            if (ea < 0) {
                const int S = lvl == 2 ? 32 : 8;
                const int bx = X.to_boundary(S, g.R), by = Y.to_boundary(S, g.R), bz = Z.to_boundary(S, g.R);
                const float inf = __int_as_float(0x7f800000);
                const float Tx = bx < 0 ? inf : time_after(X, bx), Ty = by < 0 ? inf : time_after(Y, by),
                            Tz = bz < 0 ? inf : time_after(Z, bz);
                Te = Tz, ea = 2, left = bz;
                if (Ty < Te) Te = Ty, ea = 1, left = by;
                if (Tx < Te) Te = Tx, ea = 0, left = bx;
                stuck = bx < 0 && by < 0 && bz < 0;
                fast = !stuck && Te < exitT;
                // the walk ends inside this block: nothing can be hit there
                if (!stuck && !fast) state = kMiss;
            } else {
                Te = time_after(ea == 0 ? X : (ea == 1 ? Y : Z), left);
            }
        }
        __syncwarp();
        if (fast) {
            // that axis takes this event as well, the other two, first in (x,
            // y, z), their events before it: y before x and z before both at
            // equal times
            Moment A = ea == 0 ? Y : X, B = ea == 2 ? Y : Z;
            const int na = pass(A, Te, ea == 0, max_steps), nb = pass(B, Te, ea != 2, max_steps);
            const int nx = ea == 0 ? left + 1 : na, ny = ea == 1 ? left + 1 : (ea == 0 ? na : nb),
                      nz = ea == 2 ? left + 1 : nb;
            X.tn = ea == 0 ? Te + X.ts : A.tn;
            Y.tn = ea == 1 ? Te + Y.ts : (ea == 0 ? A.tn : B.tn);
            Z.tn = ea == 2 ? Te + Z.ts : B.tn;
            X.took(nx);
            Y.took(ny);
            Z.took(nz);
            steps += nx + ny + nz;
            if (steps > max_steps) state = kMiss;
            t = Te;
            lvl = empty_level(flags, g, X.c, Y.c, Z.c);
        }
        // voxel by voxel
        __syncwarp();
        bool more = state == kWalk && (lvl == 0 || stuck);
        while (more) {
            if (++steps > max_steps) {
                state = kMiss;
                break;
            }
            float value = 1.0f;
            if (lvl == 0) {
                const size_t off = (size_t)X.c + (size_t)Y.c * R + (size_t)Z.c * RR;
                if (off >= nvox) {
                    state = kMiss;
                    break;
                }
                value = __ldg(gx + 2 * off);
            }
            at_x = X.n; at_y = Y.n; at_z = Z.n;
            // one event of the reference's walk (x when tnx < tny and tnx < tnz,
            // y when tny <= tnx and tny < tnz, else z)
            const int ox = X.c, oy = Y.c, oz = Z.c;
            const bool ex = X.tn < Y.tn && X.tn < Z.tn, ey = !(X.tn < Y.tn) && Y.tn < Z.tn;
            t = ex ? X.tn : (ey ? Y.tn : Z.tn);
            X.step(ex);
            Y.step(ey);
            Z.step(!ex && !ey);
            if (((ox ^ X.c) | (oy ^ Y.c) | (oz ^ Z.c)) >> 3) lvl = empty_level(flags, g, X.c, Y.c, Z.c);
            if (value < 0.0f) {
                state = kFine;
                break;
            }
            if (!(t < exitT)) state = kMiss;
            more = state == kWalk && lvl == 0;
        }
    }
    return state == kHit;
}

// rayCastVoxelsKernel (VoxelGrid_cuda.cu:734-770) with initRay (118-141) and
// intersectVoxelGridCuda (144-163); g.T = camera -> world
__global__ void __launch_bounds__(kRayTileX * kRayTileY, kRayCtas)
    k_raycast(const float2 *__restrict__ grid, const uint8_t *__restrict__ flags, Geom g, int iter,
              float4 *__restrict__ xyz) {
    const int xi = blockIdx.x * kRayTileX + (threadIdx.x % kRayTileX);
    const int yi = blockIdx.y * kRayTileY + (threadIdx.x / kRayTileX);
    const bool inside = xi < g.W && yi < g.H;
    const float pdx = (float)xi / g.Wf, pdy = (float)yi / g.Hf;
    float cx = -(pdx - g.K2) / g.K0, cy = -(pdy - g.K5) / g.K4, cz = -1;
    float len = 0.0f;
    len += cx * cx;
    len += cy * cy;
    len += cz * cz;
    len = 1.0f / sqrtf(len);
    cx *= len;
    cy *= len;
    cz *= len;
    Ray r;
    r.dx = g.T[0] * cx + g.T[1] * cy + g.T[2] * cz;
    r.dy = g.T[4] * cx + g.T[5] * cy + g.T[6] * cz;
    r.dz = g.T[8] * cx + g.T[9] * cy + g.T[10] * cz;
    r.ox = g.T[3];
    r.oy = g.T[7];
    r.oz = g.T[11];
    const int s0 = r.dx < 0, s1 = r.dy < 0, s2 = r.dz < 0;
    const float idx = (fabsf(r.dx) > 1e-6f) ? 1.0f / r.dx : (float)(1 - 2 * s0) * FLT_MAX;
    const float idy = (fabsf(r.dy) > 1e-6f) ? 1.0f / r.dy : (float)(1 - 2 * s1) * FLT_MAX;
    const float idz = (fabsf(r.dz) > 1e-6f) ? 1.0f / r.dz : (float)(1 - 2 * s2) * FLT_MAX;
    const float x0 = ((s0 ? g.b1x : g.b0x) - r.ox) * idx, x1 = ((s0 ? g.b0x : g.b1x) - r.ox) * idx;
    const float y0 = ((s1 ? g.b1y : g.b0y) - r.oy) * idy, y1 = ((s1 ? g.b0y : g.b1y) - r.oy) * idy;
    const float z0 = ((s2 ? g.b1z : g.b0z) - r.oz) * idz, z1 = ((s2 ? g.b0z : g.b1z) - r.oz) * idz;
    const float tmin = fmaxf(x0, fmaxf(y0, z0));
    const float tmax = fminf(x1, fminf(y1, z1));
    float4 out = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float th;
    if (traverse(inside && !(tmin >= tmax || tmax <= 0), grid, flags, g, r, idx, idy, idz, s0, s1, s2, tmin, tmax, iter,
                 &th))
        out = make_float4(th * cx, th * cy, th * cz, (th > g.min_dist && th < g.max_dist) ? 1.0f : 0.0f);
    if (inside) xyz[(size_t)yi * g.W + xi] = out;
}

// shadingKernel (VoxelGrid_cuda.cu:844-891) with filter3 (772-789)
__global__ void k_shade(const float4 *__restrict__ xyz, int W, int H, float4 *__restrict__ shaded,
                        float4 *__restrict__ normal) {
    const int xi = blockIdx.x * blockDim.x + threadIdx.x, yi = blockIdx.y * blockDim.y + threadIdx.y;
    if (xi >= W || yi >= H) return;
    const size_t off = (size_t)yi * W + xi;
    float4 pix = make_float4(0.0f, 0.0f, 0.0f, 1.0f), nrm = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (xi < W - 3 && yi < H - 3 && xi >= 3 && yi >= 3) {
        const float4 p1x = xyz[off + 1], p0x = xyz[off - 1], p1y = xyz[off + W], p0y = xyz[off - W];
        if (p1x.w > 0.0f && p0x.w > 0.0f && p1y.w > 0.0f && p0y.w > 0.0f) {
            const float ux = p1x.x - p0x.x, uy = p1x.y - p0x.y, uz = p1x.z - p0x.z;
            const float vx = p0y.x - p1y.x, vy = p0y.y - p1y.y, vz = p0y.z - p1y.z;
            float nx = uy * vz - uz * vy;
            float ny = -(ux * vz - uz * vx);
            float nz = ux * vy - uy * vx;
            float len = 0.0f;
            len += nx * nx;
            len += ny * ny;
            len += nz * nz;
            len = 1.0f / sqrtf(len);
            nx *= len;
            ny *= len;
            nz *= len;
            const float color = nx * 0.0f + ny * 0.0f + nz * 1.0f;
            if (color > 0.0f) {
                pix = make_float4(color, color, color, 1.0f);
                nrm = make_float4(nx, ny, nz, 0.0f);
            }
        }
    }
    shaded[off] = pix;
    normal[off] = nrm;
}

// ------------------------------------------------- grid and measurement --

// resetKernel (VoxelGrid_cuda.cu:113-118) with (1, 0): two voxels per store
__global__ void k_reset(float4 *__restrict__ grid2, size_t n2) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n2; i += (size_t)gridDim.x * blockDim.x)
        grid2[i] = make_float4(1.0f, 0.0f, 1.0f, 0.0f);
}

// the brick bytes of a grid given as a whole (after a copy-in or a resample)
__global__ void k_flags(const float2 *__restrict__ grid, uint8_t *__restrict__ flags, Geom g) {
    const size_t n = (size_t)g.R * g.R * g.R;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        if (grid[i].x < 0.0f) {
            const unsigned x = (unsigned)(i % g.R), y = (unsigned)((i / g.R) % g.R), z = (unsigned)(i / ((size_t)g.R * g.R));
            mark_negative(flags, g, x, y, z);
        }
}

// reconstructionKernel (VoxelGrid_cuda.cu:1090-1112): rows of the RGB-D
// frame are stored bottom-up
__global__ void k_dist_rgbd(const float4 *__restrict__ rgbd, int W, int H, float min_dist, float max_dist,
                            float *__restrict__ dist) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= W || y >= H) return;
    const float tol = 1e-4f;
    const float w = rgbd[(size_t)(H - 1 - y) * W + x].w;
    dist[(size_t)y * W + x] = (w > tol && w < (1.0f - tol)) ? w * (max_dist - min_dist) + min_dist : 0.0f;
}

__global__ void k_dist_depth16(const uint16_t *__restrict__ depth, size_t n, float *__restrict__ dist) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        dist[i] = (float)depth[i];
}

// resampleVoxelsKernel (VoxelGrid_cuda.cu:896-941); g.T = camera -> world
__global__ void k_resample(float2 *__restrict__ dst, const float2 *__restrict__ src, Geom g) {
    const int ix = blockIdx.x * blockDim.x + threadIdx.x, iy = blockIdx.y, iz = blockIdx.z;
    if (ix >= g.R) return;
    const float px = g.sx + (float)ix * g.vx2, py = g.sy + (float)iy * g.vy2, pz = g.sz + (float)iz * g.vz2;
    const float rx = g.T[0] * px + g.T[1] * py + g.T[2] * pz + g.T[3];
    const float ry = g.T[4] * px + g.T[5] * py + g.T[6] * pz + g.T[7];
    const float rz = g.T[8] * px + g.T[9] * py + g.T[10] * pz + g.T[11];
    const float qx = (rx - g.sx) / g.vx2, qy = (ry - g.sy) / g.vy2, qz = (rz - g.sz) / g.vz2;
    const float hi = (float)(g.R - 2);
    const bool oob = (qx < 0 || qx > hi) || (qy < 0 || qy > hi) || (qz < 0 || qz > hi);
    float2 v = make_float2(1.0f, 0.0f);
    float d, w;
    if (!oob && trilinear(src, g, qx, qy, qz, 0, &d) && trilinear(src, g, qx, qy, qz, 1, &w)) v = make_float2(d, w);
    dst[((size_t)iz * g.R + iy) * g.R + ix] = v;
}

}  // namespace tsdf

// ================================================================= host ==

using namespace tsdf;

struct recon_tsdf {
    recon_tsdf_params p{};
    int device = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    float2 *grid = nullptr;
    uint8_t *flags = nullptr;
    float *dist = nullptr;
    float *far_tiles = nullptr;  // of an update: the largest distance per tile of the map,
    int *list = nullptr;         // and the blocks to visit, after their number and that of those taken
    float4 *xyz = nullptr, *shaded = nullptr, *normal = nullptr;
    void *staging = nullptr;  // device copy of a host measurement (uint16 or float4 frame)
    size_t staging_bytes = 0;
    unsigned long long *counts = nullptr;
    bool counting = false;
    bool timing = false;
    double ms[kKinds] = {};
    int64_t launches[kKinds] = {};
    std::vector<std::pair<int, std::pair<cudaEvent_t, cudaEvent_t>>> pending;
    std::vector<cudaEvent_t> spare;
};

namespace {

int fail(int code, const char *msg) {
    rt::set_last_error(msg);
    return code;
}

int cuda_fail(cudaError_t e, const char *where) {
    std::string m = std::string(where) + ": " + cudaGetErrorString(e);
    rt::set_last_error(m.c_str());
    return RECON_ERR_CUDA;
}

#define TCK(call)                                            \
    do {                                                     \
        cudaError_t e_ = (call);                             \
        if (e_ != cudaSuccess) return cuda_fail(e_, #call);  \
    } while (0)

size_t n_voxels(const recon_tsdf_params &p) {
    return (size_t)p.grid_resolution * p.grid_resolution * p.grid_resolution;
}
size_t n_bricks(const recon_tsdf_params &p) {
    const size_t b = (size_t)p.grid_resolution / kBrick;
    return b * b * b;
}
// the flag bytes: one per 8^3 brick, then one per 32^3 super brick
size_t n_flag_bytes(const recon_tsdf_params &p) {
    const size_t sb = ((size_t)p.grid_resolution + 31) / 32;
    return n_bricks(p) + sb * sb * sb;
}
size_t n_pixels(const recon_tsdf_params &p) { return (size_t)p.width * p.height; }
size_t n_blocks(const recon_tsdf_params &p) {
    const size_t R = p.grid_resolution;
    return (R + kTileX - 1) / kTileX * (R / kTileY) * (R / kRunZ);
}
size_t n_far_tiles(const recon_tsdf_params &p) {
    return (size_t)((p.width + kFarTile - 1) / kFarTile) * ((p.height + kFarTile - 1) / kFarTile);
}

// invertRT4 (basic_math.cpp:355-368): VoxelGrid::setCameraParams's world ->
// camera pose, in float, translation summed left to right
void invert_rt4(const float *M, float *Mi) {
    Mi[0] = M[0]; Mi[1] = M[4]; Mi[2] = M[8];
    Mi[3] = -(M[0] * M[3] + M[4] * M[7] + M[8] * M[11]);
    Mi[4] = M[1]; Mi[5] = M[5]; Mi[6] = M[9];
    Mi[7] = -(M[1] * M[3] + M[5] * M[7] + M[9] * M[11]);
    Mi[8] = M[2]; Mi[9] = M[6]; Mi[10] = M[10];
    Mi[11] = -(M[2] * M[3] + M[6] * M[7] + M[10] * M[11]);
    Mi[12] = 0; Mi[13] = 0; Mi[14] = 0; Mi[15] = 1;
}

// whether start + n * step is exact in float for every start on the axis' grid
// (b0 + v * step) and every n that a walk of max_steps can take: b0 and step
// are multiples of a power of two u, and the sums stay below 2^24 u
bool walk_is_exact(float b0, float step, int R) {
    if (!(std::fabs(b0) < 1e30f) || !(step > 1e-30f && step < 1e30f)) return false;
    const auto unit = [](float v) {  // the exponent of the lowest bit set
        int e;
        int m = (int)std::ldexp(std::frexp(v, &e), 24);
        for (e -= 24; !(m & 1); m >>= 1) e++;
        return e;
    };
    const int u = b0 == 0.0f ? unit(step) : std::min(unit(std::fabs(b0)), unit(step));
    return std::ldexp(std::fabs((double)b0) + (double)step * (4 * R + 32), -u) < 16777216.0;
}

// the launch constants of SimParams (VoxelGrid.cpp:48-106; kernel prologues
// VoxelGrid_cuda.cu:745-756, 957-965): T3x4 is the first three rows of the
// pose the kernel uses
Geom make_geom(const recon_tsdf_params &p, const float *T3x4, const float *K) {
    Geom g;
    memset(&g, 0, sizeof(g));
    const int R = p.grid_resolution;
    g.R = R;
    g.B = R / kBrick;
    g.SB = (R + 31) / 32;
    g.nb = g.B * g.B * g.B;
    g.tiles_x = (p.width + kFarTile - 1) / kFarTile;
    g.tiles_y = (p.height + kFarTile - 1) / kFarTile;
    g.W = p.width;
    g.H = p.height;
    if (T3x4) memcpy(g.T, T3x4, sizeof(g.T));
    if (K) {
        g.K0 = K[0];
        g.K2 = K[2];
        g.K4 = K[4];
        g.K5 = K[5];
    }
    g.Wf = (float)p.width;
    g.Hf = (float)p.height;
    g.Wm2 = (float)(p.width - 2);
    g.Hm2 = (float)(p.height - 2);
    const float vsx = p.cube_dim[0] / (float)R, vsy = p.cube_dim[1] / (float)R, vsz = p.cube_dim[2] / (float)R;
    g.sx = p.cube_origin[0] - p.cube_dim[0] + vsx;
    g.sy = p.cube_origin[1] - p.cube_dim[1] + vsy;
    g.sz = p.cube_origin[2] - p.cube_dim[2] + vsz;
    g.vx2 = vsx * 2;
    g.vy2 = vsy * 2;
    g.vz2 = vsz * 2;
    g.lim = vsx * 2;
    g.tol = p.cube_dim[0] / 200.0f;
    g.slope = p.cube_dim[0] * 0.030f;
    g.inv_slope = 1.0f / g.slope;
    g.slope_lo = g.slope >= 0x1p-60f && g.slope <= 0x1p60f ? 0x1p-60f : INFINITY;
    g.b0x = p.cube_origin[0] - p.cube_dim[0];
    g.b0y = p.cube_origin[1] - p.cube_dim[1];
    g.b0z = p.cube_origin[2] - p.cube_dim[2];
    g.b1x = p.cube_origin[0] + p.cube_dim[0];
    g.b1y = p.cube_origin[1] + p.cube_dim[1];
    g.b1z = p.cube_origin[2] + p.cube_dim[2];
    g.ib0x = g.b0x + vsx;
    g.ib0y = g.b0y + vsy;
    g.ib0z = g.b0z + vsz;
    // 2.0f * voxelSize (VoxelGrid_cuda.cu:753) equals vs * 2
    g.ivx = 1.0f / g.vx2;
    g.ivy = 1.0f / g.vy2;
    g.ivz = 1.0f / g.vz2;
    g.min_dist = p.min_dist;
    g.max_dist = p.max_dist;
    for (g.mirror = 31; g.mirror < R - 1;) g.mirror = 2 * g.mirror + 1;
    g.exact_walk =
        walk_is_exact(g.ib0x, g.vx2, R) && walk_is_exact(g.ib0y, g.vy2, R) && walk_is_exact(g.ib0z, g.vz2, R);
    return g;
}

struct Timed {
    recon_tsdf *v;
    int kind;
    cudaEvent_t a = nullptr, b = nullptr;
    Timed(recon_tsdf *v_, int kind_) : v(v_), kind(kind_) {
        if (!v->timing) return;
        for (cudaEvent_t *e : {&a, &b}) {
            if (!v->spare.empty()) {
                *e = v->spare.back();
                v->spare.pop_back();
            } else if (cudaEventCreate(e) != cudaSuccess) {
                *e = nullptr;
            }
        }
        if (a) cudaEventRecord(a, v->stream);
    }
    ~Timed() {
        if (!v->timing || !a || !b) return;
        cudaEventRecord(b, v->stream);
        v->pending.push_back({kind, {a, b}});
    }
};

// A programmatic dependent of the launch before it in the stream: it may start
// while that one ends, and waits for it by itself (wait_before).
template <typename... KArgs, typename... Args>
int launch_after(void (*kern)(KArgs...), dim3 grid, dim3 block, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
    if (e != cudaSuccess) return cuda_fail(e, "kernel launch");
    rt::add_launches(1);
    return RECON_OK;
}

// Launches through cudaLaunchKernelEx, whose return value is the launch's own
// status: an error another part of the process left pending is neither
// reported as this library's nor cleared.
template <typename... KArgs, typename... Args>
int launch(void (*kern)(KArgs...), dim3 grid, dim3 block, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = s;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
    if (e != cudaSuccess) return cuda_fail(e, "kernel launch");
    rt::add_launches(1);
    return RECON_OK;
}

int check_pose(const float *T, const float *K) {
    if (!T) return fail(RECON_ERR_INVALID_ARG, "pose is NULL");
    for (int i = 0; i < 16; i++)
        if (!std::isfinite(T[i])) return fail(RECON_ERR_INVALID_ARG, "pose is not finite");
    if (K) {
        for (int i = 0; i < 9; i++)
            if (!std::isfinite(K[i])) return fail(RECON_ERR_INVALID_ARG, "K is not finite");
        if (K[0] == 0.0f || K[4] == 0.0f) return fail(RECON_ERR_INVALID_ARG, "K has a zero focal length");
    }
    return RECON_OK;
}

int ensure_staging(recon_tsdf *v, size_t bytes) {
    if (v->staging_bytes >= bytes) return RECON_OK;
    if (v->staging) {
        TCK(cudaStreamSynchronize(v->stream));
        cudaFree(v->staging);
        v->staging = nullptr;
        v->staging_bytes = 0;
    }
    TCK(cudaMalloc(&v->staging, bytes));
    v->staging_bytes = bytes;
    return RECON_OK;
}

int rebuild_flags(recon_tsdf *v, float2 *grid, uint8_t *flags) {
    TCK(cudaMemsetAsync(flags, 0, n_flag_bytes(v->p), v->stream));
    Geom g = make_geom(v->p, nullptr, nullptr);
    return launch(k_flags, dim3(1216), dim3(256), v->stream, grid, flags, g);
}

}  // namespace

extern "C" {

void recon_tsdf_default_params(int32_t grid_resolution, int32_t width, int32_t height, float min_dist,
                               float max_dist, recon_tsdf_params *out) {
    if (!out) return;
    memset(out, 0, sizeof(*out));
    out->grid_resolution = grid_resolution;
    out->cube_origin[0] = 0.0f;
    out->cube_origin[1] = 0.01f;
    out->cube_origin[2] = -1600.01f;
    out->cube_dim[0] = out->cube_dim[1] = out->cube_dim[2] = 1500.0f;
    out->width = width;
    out->height = height;
    out->min_dist = min_dist;
    out->max_dist = max_dist;
}

int recon_tsdf_create(const recon_tsdf_params *p, void *stream, recon_tsdf **out) {
    if (!p || !out) return fail(RECON_ERR_INVALID_ARG, "NULL argument");
    *out = nullptr;
    const int R = p->grid_resolution;
    if (R < 8 || R % kBrick || R > 2048) return fail(RECON_ERR_INVALID_ARG, "grid_resolution must be a multiple of 8 in 8..2048");
    if (p->width < 8 || p->height < 8 || p->width > 16384 || p->height > 16384)
        return fail(RECON_ERR_INVALID_ARG, "image size must be 8..16384");
    for (int i = 0; i < 3; i++) {
        if (!(p->cube_dim[i] > 0.0f) || !std::isfinite(p->cube_dim[i]) || !std::isfinite(p->cube_origin[i]))
            return fail(RECON_ERR_INVALID_ARG, "cube_dim must be positive and finite");
    }
    if (!(p->min_dist >= 0.0f && p->max_dist > p->min_dist)) return fail(RECON_ERR_INVALID_ARG, "need 0 <= min_dist < max_dist");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        (void)cudaGetLastError();  // this call's own error
        return fail(RECON_ERR_NO_DEVICE, "no CUDA device");
    }
    recon_tsdf *v = new recon_tsdf();
    v->p = *p;
    cudaGetDevice(&v->device);
    int rc = RECON_OK;
    auto alloc = [&](void **ptr, size_t bytes) {
        if (rc != RECON_OK) return;
        cudaError_t e = cudaMalloc(ptr, bytes);
        if (e != cudaSuccess) rc = cuda_fail(e, "cudaMalloc");
    };
    if (stream) {
        v->stream = (cudaStream_t)stream;
    } else {
        cudaError_t e = cudaStreamCreateWithFlags(&v->stream, cudaStreamNonBlocking);
        if (e != cudaSuccess) rc = cuda_fail(e, "cudaStreamCreate");
        v->own_stream = rc == RECON_OK;
    }
    alloc((void **)&v->grid, n_voxels(*p) * sizeof(float2));
    alloc((void **)&v->flags, n_flag_bytes(*p));
    alloc((void **)&v->dist, n_pixels(*p) * sizeof(float));
    alloc((void **)&v->far_tiles, n_far_tiles(*p) * sizeof(float));
    alloc((void **)&v->list, (2 + n_blocks(*p)) * sizeof(int));
    alloc((void **)&v->xyz, n_pixels(*p) * sizeof(float4));
    alloc((void **)&v->shaded, n_pixels(*p) * sizeof(float4));
    alloc((void **)&v->normal, n_pixels(*p) * sizeof(float4));
    alloc((void **)&v->counts, 4 * sizeof(unsigned long long));
    if (rc == RECON_OK) {
        cudaMemsetAsync(v->dist, 0, n_pixels(*p) * sizeof(float), v->stream);
        cudaMemsetAsync(v->xyz, 0, n_pixels(*p) * sizeof(float4), v->stream);
        cudaMemsetAsync(v->shaded, 0, n_pixels(*p) * sizeof(float4), v->stream);
        cudaMemsetAsync(v->normal, 0, n_pixels(*p) * sizeof(float4), v->stream);
        cudaMemsetAsync(v->counts, 0, 4 * sizeof(unsigned long long), v->stream);
        rc = recon_tsdf_reset(v);
    }
    if (rc != RECON_OK) {
        recon_tsdf_destroy(v);
        return rc;
    }
    *out = v;
    return RECON_OK;
}

int recon_tsdf_destroy(recon_tsdf *v) {
    if (!v) return RECON_OK;
    if (v->stream) cudaStreamSynchronize(v->stream);
    for (auto &pe : v->pending) {
        cudaEventDestroy(pe.second.first);
        cudaEventDestroy(pe.second.second);
    }
    for (cudaEvent_t e : v->spare) cudaEventDestroy(e);
    cudaFree(v->grid);
    cudaFree(v->flags);
    cudaFree(v->dist);
    cudaFree(v->far_tiles);
    cudaFree(v->list);
    cudaFree(v->xyz);
    cudaFree(v->shaded);
    cudaFree(v->normal);
    cudaFree(v->staging);
    cudaFree(v->counts);
    if (v->own_stream) cudaStreamDestroy(v->stream);
    delete v;
    return RECON_OK;
}

int recon_tsdf_reset(recon_tsdf *v) {
    if (!v) return fail(RECON_ERR_INVALID_ARG, "NULL grid");
    Timed tm(v, 4);
    TCK(cudaMemsetAsync(v->flags, 0, n_flag_bytes(v->p), v->stream));
    return launch(k_reset, dim3(152 * 8), dim3(256), v->stream, reinterpret_cast<float4 *>(v->grid), n_voxels(v->p) / 2);
}

int recon_tsdf_set_dist_map(recon_tsdf *v, const float *dist, int32_t on_device) {
    if (!v || !dist) return fail(RECON_ERR_INVALID_ARG, "NULL argument");
    TCK(cudaMemcpyAsync(v->dist, dist, n_pixels(v->p) * sizeof(float),
                        on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, v->stream));
    return RECON_OK;
}

int recon_tsdf_set_dist_rgbd_float4(recon_tsdf *v, const float *rgbd, int32_t on_device) {
    if (!v || !rgbd) return fail(RECON_ERR_INVALID_ARG, "NULL argument");
    const float4 *src = reinterpret_cast<const float4 *>(rgbd);
    if (!on_device) {
        int rc = ensure_staging(v, n_pixels(v->p) * sizeof(float4));
        if (rc) return rc;
        TCK(cudaMemcpyAsync(v->staging, rgbd, n_pixels(v->p) * sizeof(float4), cudaMemcpyHostToDevice, v->stream));
        src = reinterpret_cast<const float4 *>(v->staging);
    }
    Timed tm(v, 3);
    dim3 blk(32, 8), grd((v->p.width + 31) / 32, (v->p.height + 7) / 8);
    return launch(k_dist_rgbd, grd, blk, v->stream, src, v->p.width, v->p.height, v->p.min_dist, v->p.max_dist, v->dist);
}

int recon_tsdf_set_dist_depth16(recon_tsdf *v, const uint16_t *depth, int32_t on_device) {
    if (!v || !depth) return fail(RECON_ERR_INVALID_ARG, "NULL argument");
    const uint16_t *src = depth;
    if (!on_device) {
        int rc = ensure_staging(v, n_pixels(v->p) * sizeof(uint16_t));
        if (rc) return rc;
        TCK(cudaMemcpyAsync(v->staging, depth, n_pixels(v->p) * sizeof(uint16_t), cudaMemcpyHostToDevice, v->stream));
        src = reinterpret_cast<const uint16_t *>(v->staging);
    }
    Timed tm(v, 3);
    return launch(k_dist_depth16, dim3((unsigned)((n_pixels(v->p) + 255) / 256)), dim3(256), v->stream, src,
                  n_pixels(v->p), v->dist);
}

int recon_tsdf_update(recon_tsdf *v, const float T[16], const float K[9]) {
    if (!v || !K) return fail(RECON_ERR_INVALID_ARG, "NULL argument");
    int rc = check_pose(T, K);
    if (rc) return rc;
    float Tin[16], Tw2c[16];
    memcpy(Tin, T, sizeof(Tin));
    invert_rt4(Tin, Tw2c);
    Geom g = make_geom(v->p, Tw2c, K);
    const int R = v->p.grid_resolution;
    dim3 grd((R + kTileX - 1) / kTileX, R / kTileY, R / kRunZ);
    Timed tm(v, 0);
    // the counts are of all voxels that project into the image, hidden ones too
    if (v->counting)
        return launch(k_update<true>, grd, dim3(kTileX * kTileY), v->stream, v->grid, v->flags, v->dist, g, v->counts);
    const int n = (int)(grd.x * grd.y * grd.z);
    if (n < kListBlocks)
        return launch(k_update<false>, grd, dim3(kTileX * kTileY), v->stream, v->grid, v->flags, v->dist, g,
                      (unsigned long long *)nullptr);
    rc = launch(k_far_tiles, dim3((g.tiles_x * g.tiles_y + 3) / 4), dim3(128), v->stream, v->dist, g, v->far_tiles, v->list);
    if (!rc)
        rc = launch_after(k_pick_blocks, dim3((n + 31) / 32), dim3(256), v->stream, v->far_tiles, g, (int)grd.x, (int)grd.y, n,
                    v->list + 2, v->list);
    if (!rc)
        rc = launch_after(k_update_list, dim3(152 * kUpdateCtas), dim3(kTileX * kTileY), v->stream, v->grid, v->flags, v->dist, g,
                    (int)grd.x, (int)grd.y, v->list + 2, v->list);
    return rc;
}

int recon_tsdf_raycast(recon_tsdf *v, const float T[16], const float K[9], int32_t cubic_filter) {
    if (!v || !K) return fail(RECON_ERR_INVALID_ARG, "NULL argument");
    int rc = check_pose(T, K);
    if (rc) return rc;
    Geom g = make_geom(v->p, T, K);
    dim3 grd((v->p.width + kRayTileX - 1) / kRayTileX, (v->p.height + kRayTileY - 1) / kRayTileY);
    {
        Timed tm(v, 1);
        rc = launch(k_raycast, grd, dim3(kRayTileX * kRayTileY), v->stream, v->grid, v->flags, g, cubic_filter ? 3 : 0,
                    v->xyz);
        if (rc) return rc;
    }
    Timed tm(v, 2);
    dim3 blk(32, 8), grd2((v->p.width + 31) / 32, (v->p.height + 7) / 8);
    return launch(k_shade, grd2, blk, v->stream, v->xyz, v->p.width, v->p.height, v->shaded, v->normal);
}

int recon_tsdf_resample(recon_tsdf *dst, recon_tsdf *src, const float T[16]) {
    if (!dst || !src || dst == src) return fail(RECON_ERR_INVALID_ARG, "need two different grids");
    if (memcmp(&dst->p, &src->p, sizeof(recon_tsdf_params)) != 0)
        return fail(RECON_ERR_INVALID_ARG, "the grids have different parameters");
    int rc = check_pose(T, nullptr);
    if (rc) return rc;
    if (src->stream != dst->stream) {
        cudaEvent_t e;
        TCK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        cudaEventRecord(e, src->stream);
        cudaStreamWaitEvent(dst->stream, e, 0);
        cudaEventDestroy(e);
    }
    Geom g = make_geom(dst->p, T, nullptr);
    const int R = dst->p.grid_resolution;
    {
        Timed tm(dst, 4);
        rc = launch(k_resample, dim3((R + 127) / 128, R, R), dim3(128), dst->stream, dst->grid, src->grid, g);
        if (rc) return rc;
    }
    rc = rebuild_flags(dst, dst->grid, dst->flags);
    if (rc) return rc;
    if (src->stream != dst->stream) {
        // src must not be changed before the resample has read it
        cudaEvent_t e;
        TCK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        cudaEventRecord(e, dst->stream);
        cudaStreamWaitEvent(src->stream, e, 0);
        cudaEventDestroy(e);
    }
    return RECON_OK;
}

void *recon_tsdf_device_array(recon_tsdf *v, const char *name) {
    if (!v || !name) return nullptr;
    if (!strcmp(name, "tsdf")) return v->grid;
    if (!strcmp(name, "dist")) return v->dist;
    if (!strcmp(name, "xyz")) return v->xyz;
    if (!strcmp(name, "shaded")) return v->shaded;
    if (!strcmp(name, "normal")) return v->normal;
    if (!strcmp(name, "flags")) return v->flags;
    return nullptr;
}

int64_t recon_tsdf_get(recon_tsdf *v, const char *name, void *host_dst, int64_t nbytes) {
    if (!v || !name || !host_dst) return fail(RECON_ERR_INVALID_ARG, "NULL argument");
    void *src = recon_tsdf_device_array(v, name);
    if (!src) return fail(RECON_ERR_INVALID_ARG, "unknown array");
    size_t bytes;
    if (!strcmp(name, "tsdf"))
        bytes = n_voxels(v->p) * sizeof(float2);
    else if (!strcmp(name, "dist"))
        bytes = n_pixels(v->p) * sizeof(float);
    else if (!strcmp(name, "flags"))
        bytes = n_bricks(v->p);
    else
        bytes = n_pixels(v->p) * sizeof(float4);
    if ((int64_t)bytes > nbytes) return fail(RECON_ERR_INVALID_ARG, "destination too small");
    TCK(cudaMemcpyAsync(host_dst, src, bytes, cudaMemcpyDeviceToHost, v->stream));
    TCK(cudaStreamSynchronize(v->stream));
    return (int64_t)bytes;
}

int recon_tsdf_set_grid(recon_tsdf *v, const float *grid, int32_t on_device) {
    if (!v || !grid) return fail(RECON_ERR_INVALID_ARG, "NULL argument");
    TCK(cudaMemcpyAsync(v->grid, grid, n_voxels(v->p) * sizeof(float2),
                        on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, v->stream));
    return rebuild_flags(v, v->grid, v->flags);
}

void *recon_tsdf_stream(recon_tsdf *v) { return v ? (void *)v->stream : nullptr; }

int recon_tsdf_enable_timing(recon_tsdf *v, int32_t on) {
    if (!v) return fail(RECON_ERR_INVALID_ARG, "NULL grid");
    v->timing = on != 0;
    return RECON_OK;
}

int recon_tsdf_get_timing(recon_tsdf *v, double ms[5], int64_t launches[5], int32_t reset) {
    if (!v) return fail(RECON_ERR_INVALID_ARG, "NULL grid");
    TCK(cudaStreamSynchronize(v->stream));
    for (auto &pe : v->pending) {
        float t = 0.0f;
        if (cudaEventElapsedTime(&t, pe.second.first, pe.second.second) == cudaSuccess) {
            v->ms[pe.first] += t;
            v->launches[pe.first] += 1;
        }
        v->spare.push_back(pe.second.first);
        v->spare.push_back(pe.second.second);
    }
    v->pending.clear();
    for (int k = 0; k < kKinds; k++) {
        if (ms) ms[k] = v->ms[k];
        if (launches) launches[k] = v->launches[k];
        if (reset) {
            v->ms[k] = 0.0;
            v->launches[k] = 0;
        }
    }
    return RECON_OK;
}

int recon_tsdf_enable_counting(recon_tsdf *v, int32_t on) {
    if (!v) return fail(RECON_ERR_INVALID_ARG, "NULL grid");
    v->counting = on != 0;
    return RECON_OK;
}

int recon_tsdf_get_counts(recon_tsdf *v, int64_t counts[3], int32_t reset) {
    if (!v || !counts) return fail(RECON_ERR_INVALID_ARG, "NULL argument");
    unsigned long long h[4];
    TCK(cudaMemcpyAsync(h, v->counts, sizeof(h), cudaMemcpyDeviceToHost, v->stream));
    TCK(cudaStreamSynchronize(v->stream));
    for (int i = 0; i < 3; i++) counts[i] = (int64_t)h[i];
    if (reset) TCK(cudaMemsetAsync(v->counts, 0, sizeof(h), v->stream));
    return RECON_OK;
}

}  // extern "C"
