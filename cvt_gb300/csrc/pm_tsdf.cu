/*
 * pm_tsdf.cu — TSDF fusion of depth maps (the consumer of the disparity maps):
 * cvt::TSDFVolume (cvt/vision/TSDFVolume.h, TSDFVolume.cpp) with the kernels
 * of cvt/cl/kernel/TSDFVolume/TSDFVolume.cl.
 *
 *   k_tsdf_clear    TSDFVolume_clear:  every voxel (1, weight)
 *   k_tsdf_add      TSDFVolume_add:    project the voxel with TG2CAM = proj *
 *                   grid-to-world, read the depth map at the nearest texel and
 *                   fold the truncated signed distance into a running mean
 *   k_tsdf_raycast  TSDFVolume_rayCastDepthmap: march each pixel's ray through
 *                   the volume (half a voxel along its dominant axis) with
 *                   trilinear reads and report the depth of the first + to -
 *                   crossing
 *   k_tsdf_slice    TSDFVolume_sliceX/Y/Z (the reference's host wrappers are
 *                   empty; the kernels' arithmetic is given here)
 *
 * The volume is W*H*D float2 (tsdf, weight), x fastest (TSDFVolume.cpp:38).
 * Matrices are row-major 4x4, as the kernels' Mat4f (cvt/cl/kernel/Matrix4.cl)
 * and cvt::Matrix4f store them.  Host matrix products follow Matrix4.h:269-288
 * (left-to-right sums) and the inverse Matrix.cpp:109-196 (cofactors; a
 * matrix with |det| < FLT_EPSILON is returned unchanged, as inverseSelf
 * leaves it).  Device arithmetic is the kernels' own, compiled without
 * contraction; OpenCL's normalize is v * (1 / sqrt(dot(v, v))) and dot is
 * summed left to right.  Clear is an HBM write stream (8 B per voxel); add
 * projects every voxel (two divisions: issue-bound) and reads and writes 16 B
 * only inside the truncation band; the ray cast is a latency-bound gather.
 *
 * The ray loop of the reference (`for (lambda = start + step; lambda <= end;
 * lambda += step)`) never ends where lambda + step rounds to lambda (a camera
 * ~2^24 voxels from the volume).  Here it stops after 2 * max(W, H, D) + 16
 * steps — more than the 2 steps per voxel along the dominant axis a ray can
 * take — and such a pixel keeps the value 0.
 */
#include <float.h>
#include <math.h>
#include <stdio.h>
#include <string.h>

#include <string>
#include <vector>

#include "cvtpm.h"
#include "cvtpm_tools.h"
#include "pm_kernels.cuh"

namespace {

struct Mat4 {
    float m[16];
};

/* Matrix4::operator* (Matrix4.h:269-288) */
Mat4 mat4_mul(const Mat4& a, const Mat4& b) {
    Mat4 r;
    for (int i = 0; i < 4; ++i)
        for (int j = 0; j < 4; ++j)
            r.m[i * 4 + j] = a.m[i * 4] * b.m[j] + a.m[i * 4 + 1] * b.m[4 + j] + a.m[i * 4 + 2] * b.m[8 + j] +
                             a.m[i * 4 + 3] * b.m[12 + j];
    return r;
}

/* Matrix4::inverseSelf (Matrix.cpp:109-196): 2x2 and 3x3 minors of the
 * Laplace expansion, in the reference's order; |det| < FLT_EPSILON leaves the
 * matrix as it is. */
Mat4 mat4_inverse(const Mat4& in) {
    const float* a = in.m;
#define M(i, j) a[(i) * 4 + (j)]
    const float d23_01 = M(2, 0) * M(3, 1) - M(3, 0) * M(2, 1), d23_02 = M(2, 0) * M(3, 2) - M(3, 0) * M(2, 2);
    const float d23_03 = M(2, 0) * M(3, 3) - M(3, 0) * M(2, 3), d23_12 = M(2, 1) * M(3, 2) - M(3, 1) * M(2, 2);
    const float d23_13 = M(2, 1) * M(3, 3) - M(3, 1) * M(2, 3), d23_23 = M(2, 2) * M(3, 3) - M(3, 2) * M(2, 3);
    const float c123_123 = M(1, 1) * d23_23 - M(1, 2) * d23_13 + M(1, 3) * d23_12;
    const float c123_023 = M(1, 0) * d23_23 - M(1, 2) * d23_03 + M(1, 3) * d23_02;
    const float c123_013 = M(1, 0) * d23_13 - M(1, 1) * d23_03 + M(1, 3) * d23_01;
    const float c123_012 = M(1, 0) * d23_12 - M(1, 1) * d23_02 + M(1, 2) * d23_01;
    const float det = M(0, 0) * c123_123 - M(0, 1) * c123_023 + M(0, 2) * c123_013 - M(0, 3) * c123_012;
    if (fabsf(det) < FLT_EPSILON) return in;
    const float inv = 1.0f / det;
    const float c023_123 = M(0, 1) * d23_23 - M(0, 2) * d23_13 + M(0, 3) * d23_12;
    const float c023_023 = M(0, 0) * d23_23 - M(0, 2) * d23_03 + M(0, 3) * d23_02;
    const float c023_013 = M(0, 0) * d23_13 - M(0, 1) * d23_03 + M(0, 3) * d23_01;
    const float c023_012 = M(0, 0) * d23_12 - M(0, 1) * d23_02 + M(0, 2) * d23_01;
    const float d13_01 = M(1, 0) * M(3, 1) - M(3, 0) * M(1, 1), d13_02 = M(1, 0) * M(3, 2) - M(3, 0) * M(1, 2);
    const float d13_03 = M(1, 0) * M(3, 3) - M(3, 0) * M(1, 3), d13_12 = M(1, 1) * M(3, 2) - M(3, 1) * M(1, 2);
    const float d13_13 = M(1, 1) * M(3, 3) - M(3, 1) * M(1, 3), d13_23 = M(1, 2) * M(3, 3) - M(3, 2) * M(1, 3);
    const float c013_123 = M(0, 1) * d13_23 - M(0, 2) * d13_13 + M(0, 3) * d13_12;
    const float c013_023 = M(0, 0) * d13_23 - M(0, 2) * d13_03 + M(0, 3) * d13_02;
    const float c013_013 = M(0, 0) * d13_13 - M(0, 1) * d13_03 + M(0, 3) * d13_01;
    const float c013_012 = M(0, 0) * d13_12 - M(0, 1) * d13_02 + M(0, 2) * d13_01;
    const float d12_01 = M(1, 0) * M(2, 1) - M(2, 0) * M(1, 1), d12_02 = M(1, 0) * M(2, 2) - M(2, 0) * M(1, 2);
    const float d12_03 = M(1, 0) * M(2, 3) - M(2, 0) * M(1, 3), d12_12 = M(1, 1) * M(2, 2) - M(2, 1) * M(1, 2);
    const float d12_13 = M(1, 1) * M(2, 3) - M(2, 1) * M(1, 3), d12_23 = M(1, 2) * M(2, 3) - M(2, 2) * M(1, 3);
    const float c012_123 = M(0, 1) * d12_23 - M(0, 2) * d12_13 + M(0, 3) * d12_12;
    const float c012_023 = M(0, 0) * d12_23 - M(0, 2) * d12_03 + M(0, 3) * d12_02;
    const float c012_013 = M(0, 0) * d12_13 - M(0, 1) * d12_03 + M(0, 3) * d12_01;
    const float c012_012 = M(0, 0) * d12_12 - M(0, 1) * d12_02 + M(0, 2) * d12_01;
#undef M
    const Mat4 r = {{c123_123 * inv, -c023_123 * inv, c013_123 * inv, -c012_123 * inv,
                     -c123_023 * inv, c023_023 * inv, -c013_023 * inv, c012_023 * inv,
                     c123_013 * inv, -c023_013 * inv, c013_013 * inv, -c012_013 * inv,
                     -c123_012 * inv, c023_012 * inv, -c013_012 * inv, c012_012 * inv}};
    return r;
}

/* ------------------------------------------------------------ device -- */
struct DMat4 {
    float4 r[4];
};

DMat4 to_dev(const Mat4& a) {
    DMat4 d;
    for (int i = 0; i < 4; ++i) d.r[i] = make_float4(a.m[i * 4], a.m[i * 4 + 1], a.m[i * 4 + 2], a.m[i * 4 + 3]);
    return d;
}

/* dot4 (pm_device.cuh) sums left to right, as OpenCL's dot is emulated */
__device__ __forceinline__ float4 xform(const DMat4& m, float4 v) {   /* mat4f_transform (Matrix4.cl) */
    return make_float4(dot4(m.r[0], v), dot4(m.r[1], v), dot4(m.r[2], v), dot4(m.r[3], v));
}
__device__ __forceinline__ float mixf(float a, float b, float t) { return a + (b - a) * t; }

/* clear: two voxels per 16-byte store over the linear volume (512^3: 0.141 ms
 * = 7.6 TB/s, against 0.267 ms with one 8-byte store per voxel).  add:
 * TSDF_ZPT z-planes per thread (512^3, 640x480 map: 1 plane 0.310 ms, 2 0.306,
 * 4 0.249, 8 0.220). */
#define TSDF_CLEAR_VEC 1
#define TSDF_ZPT 8
__global__ void __launch_bounds__(256) k_tsdf_clear(float2* __restrict__ cv, int W, int H, int D, float init) {
    const int x = blockIdx.x * 32 + threadIdx.x, y = blockIdx.y * 8 + threadIdx.y, z = blockIdx.z;
    if (x >= W || y >= H || z >= D) return;
    cv[((size_t)z * H + y) * W + x] = make_float2(1.0f, init);
}

/* The same over the volume as n voxels: thread i writes voxels 2i and 2i+1
 * with one 16-byte store (the allocation is 256-byte aligned). */
__global__ void __launch_bounds__(256) k_tsdf_clear_vec(float4* __restrict__ cv4, size_t n, float init) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (2 * i + 1 < n) cv4[i] = make_float4(1.0f, init, 1.0f, init);
    else if (2 * i < n) ((float2*)cv4)[2 * i] = make_float2(1.0f, init);
}

__device__ __forceinline__ void tsdf_add_voxel(float2* __restrict__ cv, int W, int H, int x, int y, int z,
                                               const float* __restrict__ dmap, size_t dpitch4, int iw, int ih,
                                               float dscale, const DMat4& tg2cam, float trunc) {
    const float4 g = xform(tg2cam, make_float4((float)x, (float)y, (float)z, 1.0f));
    /* Voxels the update would skip anyway, found without the two divisions:
     * it needs g.z > 0 (the depth read before that test has no effect), and
     * for g.z > 0 a numerator beyond -2 g.z or (size + 2) g.z makes the
     * rounded quotient < 0 or > size (the product rounds by at most one part
     * in 2^24).  NaN and infinite values fall through to the full test. */
    if (!(g.z > 0.0f)) return;
    const float lo = -2.0f * g.z;
    if (g.x < lo || g.y < lo || g.x > ((float)iw + 2.0f) * g.z || g.y > ((float)ih + 2.0f) * g.z) return;
    const float ix = g.x / g.z, iy = g.y / g.z;
    if (ix < (float)iw && iy < (float)ih && ix >= 0.0f && iy >= 0.0f) {
        const float d = dmap[(size_t)(int)floorf(iy) * dpitch4 + (int)floorf(ix)] * dscale;   /* nearest texel */
        if (d > 0.0f && g.z > 0.0f) {
            const float sdf = d - g.z, w = 1.0f;
            const float tsdf = sdf / trunc;
            if (fabsf(sdf) <= trunc) {
                float2* p = cv + ((size_t)z * H + y) * W + x;
                const float2 o = *p;
                *p = make_float2((o.x * o.y + tsdf * w) / (o.y + w), o.y + w);
            }
        }
    }
}

__global__ void __launch_bounds__(256) k_tsdf_add(float2* __restrict__ cv, int W, int H, int D,
                                                  const float* __restrict__ dmap, size_t dpitch4, int iw, int ih,
                                                  float dscale, DMat4 tg2cam, float trunc) {
    const int x = blockIdx.x * 32 + threadIdx.x, y = blockIdx.y * 8 + threadIdx.y;
    if (x >= W || y >= H) return;
#pragma unroll 1
    for (int z = blockIdx.z * TSDF_ZPT; z < min(D, (int)(blockIdx.z + 1) * TSDF_ZPT); ++z)
        tsdf_add_voxel(cv, W, H, x, y, z, dmap, dpitch4, iw, ih, dscale, tg2cam, trunc);
}

/* TSDFVolume_trilinearValue: 1e10 if a corner has weight < 1 */
__device__ __forceinline__ float trilinear(const float2* __restrict__ cv, int W, int H, int D, float px, float py,
                                           float pz) {
    px = fminf(fmaxf(0.0f, px), (float)(W - 2));
    py = fminf(fmaxf(0.0f, py), (float)(H - 2));
    pz = fminf(fmaxf(0.0f, pz), (float)(D - 2));
    const float bx = floorf(px), by = floorf(py), bz = floorf(pz);
    const float ax = px - bx, ay = py - by, az = pz - bz;
    const int ix = (int)bx, iy = (int)by, iz = (int)bz;
    /* s0..s7: x fastest, then y, then z.  The first alone settles most empty
     * samples; the others are in flight together (a test between them would
     * make each wait for the one before). */
    const float2* const p = cv + ((size_t)iz * H + iy) * W + ix;
    const float2 t0 = __ldg(p);
    if (t0.y < 1.0f) return 1e10f;
    float2 t[8];
    float v[8];
    t[0] = t0;
#pragma unroll
    for (int k = 1; k < 8; ++k) t[k] = __ldg(p + ((size_t)(k >> 2) * H + ((k >> 1) & 1)) * W + (k & 1));
    bool seen = true;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        seen = seen && !(t[k].y < 1.0f);
        v[k] = t[k].x;
    }
    if (!seen) return 1e10f;
    const float z0 = mixf(v[0], v[4], az), z1 = mixf(v[1], v[5], az), z2 = mixf(v[2], v[6], az), z3 = mixf(v[3], v[7], az);
    const float y0 = mixf(z0, z2, ay), y1 = mixf(z1, z3, ay);
    return mixf(y0, y1, ax);
}

__device__ __forceinline__ float ray_bound(float o, float d, int extent, bool start) {
    return (((d > 0.0f) == start ? 0.0f : (float)extent) - o) / d;
}

/* Which bricks of 8^3 voxels hold a voxel of weight >= 1 (or NaN: the test of
 * trilinear, inverted), one byte each; and from those, which bricks of 32^3
 * do.  A thread reads a column of 64 voxels of one x; the volume is read once,
 * 8 bytes per voxel (HBM-bound).  The bytes are a volume's own and every cast
 * forms them anew, each byte stored once and never cleared first: casts of one
 * volume on several streams store the values that are there, so one may march
 * while another marks. */
#define TSDF_FINE 3                                  /* log2 of the extents */
#define TSDF_COARSE 5
struct BrickGrid {
    const unsigned char *fine, *coarse;              /* NULL: no bricks */
    int fw, fh, cw, ch;                              /* bricks per row and per column */
};
__global__ void __launch_bounds__(256) k_tsdf_bricks(const float2* __restrict__ cv, int W, int H, int D,
                                                     unsigned char* __restrict__ fine, BrickGrid g) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y0 = blockIdx.y * 8, z0 = blockIdx.z * 8;
    bool any = false;
    if (x < W) {
        const int y1 = min(y0 + 8, H), z1 = min(z0 + 8, D);
#pragma unroll 4
        for (int z = z0; z < z1; ++z) {
            const float2* p = cv + ((size_t)z * H + y0) * W + x;
            if (y1 == y0 + 8) {
                float w[8];
#pragma unroll
                for (int y = 0; y < 8; ++y) w[y] = __ldg(p + (size_t)y * W).y;
#pragma unroll
                for (int y = 0; y < 8; ++y) any |= !(w[y] < 1.0f);
            } else {
                for (int y = y0; y < y1; ++y, p += W) any = any || !(__ldg(p).y < 1.0f);
            }
        }
    }
    const unsigned m = __ballot_sync(0xffffffffu, any);
    if ((threadIdx.x & 7) == 0 && x < W)
        fine[((size_t)blockIdx.z * g.fh + blockIdx.y) * g.fw + (x >> 3)] = (m >> (threadIdx.x & 31)) & 0xffu ? 1 : 0;
}

/* A coarse brick per warp: any of its 4^3 fine ones (fd of them in z). */
__global__ void __launch_bounds__(256) k_tsdf_coarse(const unsigned char* __restrict__ fine, unsigned char* __restrict__ coarse,
                                                     BrickGrid g, int fd, int cd) {
    const unsigned i = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (i >= (unsigned)(g.cw * g.ch * cd)) return;
    const int cx = (int)(i % g.cw), cy = (int)(i / g.cw % g.ch), cz = (int)(i / g.cw / g.ch);
    const int x = 4 * cx + (lane & 3), y = 4 * cy + (lane >> 2 & 3), z = 4 * cz + (lane >> 4);
    bool any = false;
    if (x < g.fw && y < g.fh) {
        if (z < fd) any = fine[((size_t)z * g.fh + y) * g.fw + x];
        if (z + 2 < fd) any = any || fine[((size_t)(z + 2) * g.fh + y) * g.fw + x];
    }
    any = __any_sync(0xffffffffu, any);
    if (lane == 0) coarse[i] = any;
}

/* The march evaluates samples half a voxel apart, and most of them lie where
 * nothing was integrated: a corner of weight < 1 makes the value 1e10.  With
 * BRICKS, a sample whose first corner lies in a brick without weights has that
 * value at once.  It then steps to the last sample it expects inside the brick,
 * with the additions to lambda alone: if that one is in the brick, so are those
 * between (a position is monotone in lambda, rounded or not) and all have the
 * value 1e10; if not, it takes one step.  The values met, and so the results,
 * are those of the plain march.  That is a kernel of its own: with the bricks'
 * registers in its loop it took 10-16 % longer (256^3, 64x48 rays, empty, 0.146
 * -> 0.168 ms). */
template <bool BRICKS>
__global__ void __launch_bounds__(256) k_tsdf_raycast(float* __restrict__ out, size_t opitch4, int iw, int ih,
                                                      const float2* __restrict__ cv, int W, int H, int D,
                                                      BrickGrid bg,
                                                      DMat4 tcam2g, DMat4 tg2cam, float scale, int max_steps) {
    const int gx = blockIdx.x * 32 + threadIdx.x, gy = blockIdx.y * 8 + threadIdx.y;
    if (gx >= iw || gy >= ih) return;
    const float4 o4 = xform(tcam2g, make_float4(0.0f, 0.0f, 0.0f, 1.0f));
    const float4 t4 = xform(tcam2g, make_float4((float)gx, (float)gy, 1.0f, 1.0f));
    float dx = t4.x - o4.x, dy = t4.y - o4.y, dz = t4.z - o4.z;
    const float rn = 1.0f / sqrtf((dx * dx + dy * dy) + dz * dz);   /* normalize */
    dx = dx * rn; dy = dy * rn; dz = dz * rn;
    const float rs = fmaxf(fmaxf(ray_bound(o4.x, dx, W, true), ray_bound(o4.y, dy, H, true)), ray_bound(o4.z, dz, D, true));
    const float re = fminf(fminf(ray_bound(o4.x, dx, W, false), ray_bound(o4.y, dy, H, false)), ray_bound(o4.z, dz, D, false));
    float ret = 0.0f;
    if (rs < re && isfinite(rs) && isfinite(re) && isfinite(dx) && isfinite(dy) && isfinite(dz)) {
        const float vx = fabsf(dx * (re - rs)), vy = fabsf(dy * (re - rs)), vz = fabsf(dz * (re - rs));
        const float step = 0.5f * sqrtf((vx * vx + vy * vy) + vz * vz) / fmaxf(vx, fmaxf(vy, vz));
        float ppz = o4.z + dz * rs;
        float vp = trilinear(cv, W, H, D, o4.x + dx * rs, o4.y + dy * rs, ppz);
        int n = 0;
        float lambda = rs + step;
        /* a sample's value against the one before: true where the march ends */
        auto met = [&](float v, float pz) {
            if (vp < 0.0f && v > 0.0f) return true;
            if (vp > 0.0f && v < 0.0f) {
                const float alpha = -v / (vp - v);
                const float g = mixf(pz, ppz, alpha);   /* the reference mixes z only and uses it for x, y, z */
                ret = fmaxf(-(dot4(tg2cam.r[2], make_float4(g, g, g, 1.0f))) * scale, 0.0f);
                return true;
            }
            vp = v;
            ppz = pz;
            return false;
        };
        if (!BRICKS) {
            for (; lambda <= re && n < max_steps; lambda += step, ++n) {
                const float px = o4.x + dx * lambda, py = o4.y + dy * lambda, pz = o4.z + dz * lambda;
                if (met(trilinear(cv, W, H, D, px, py, pz), pz)) break;
            }
        } else {
            const float mx = (float)(W - 2), my = (float)(H - 2), mz = (float)(D - 2);
            /* the first corner of the sample at lambda (trilinear's clamps) */
            auto corner = [&](float lambda) {
                return make_int3((int)fminf(fmaxf(0.0f, o4.x + dx * lambda), mx), (int)fminf(fmaxf(0.0f, o4.y + dy * lambda), my),
                                 (int)fminf(fmaxf(0.0f, o4.z + dz * lambda), mz));
            };
            const float ix = 1.0f / (dx * step), iy = 1.0f / (dy * step), iz = 1.0f / (dz * step);   /* steps per voxel */
            while (lambda <= re && n < max_steps) {
                bool empty = false;
                {
                    const int3 c = corner(lambda);
                    int sh = TSDF_COARSE;
                    empty = !__ldg(&bg.coarse[((c.z >> sh) * bg.ch + (c.y >> sh)) * bg.cw + (c.x >> sh)]);
                    if (!empty) {
                        sh = TSDF_FINE;
                        empty = !__ldg(&bg.fine[((c.z >> sh) * bg.fh + (c.y >> sh)) * bg.fw + (c.x >> sh)]);
                    }
                    if (empty && !(vp < 0.0f)) {             /* 1e10 from here on makes no crossing */
                        const int3 b = make_int3(c.x >> sh, c.y >> sh, c.z >> sh);
                        /* the steps to the brick's far sides, less a little */
                        const float ex = (float)((b.x + (dx > 0.0f)) << sh) - (o4.x + dx * lambda);
                        const float ey = (float)((b.y + (dy > 0.0f)) << sh) - (o4.y + dy * lambda);
                        const float ez = (float)((b.z + (dz > 0.0f)) << sh) - (o4.z + dz * lambda);
                        const float far = fminf(fminf(dx != 0.0f ? ex * ix : 1e9f, dy != 0.0f ? ey * iy : 1e9f),
                                                dz != 0.0f ? ez * iz : 1e9f) - 0.01f;
                        const int hop = min((int)fminf(fmaxf(far, 0.0f), 256.0f), max_steps - n - 1);
                        if (hop > 0) {
                            float last = lambda;
                            for (int i = 0; i < hop; ++i) last += step;
                            const int3 l = corner(last);
                            if (last <= re && l.x >> sh == b.x && l.y >> sh == b.y && l.z >> sh == b.z) {
                                vp = 1e10f;
                                ppz = o4.z + dz * last;
                                lambda = last + step;
                                n += hop + 1;
                                continue;
                            }
                        }
                    }
                }
                const float pz = o4.z + dz * lambda;
                if (met(empty ? 1e10f : trilinear(cv, W, H, D, o4.x + dx * lambda, o4.y + dy * lambda, pz), pz)) break;
                lambda += step;
                ++n;
            }
        }
    }
    out[(size_t)gy * opitch4 + gx] = ret;
}

/* TSDFVolume_sliceX/Y/Z: RGBA (clamp(tsdf + 0.5, 0, 1) x3, 1) at plane v */
__global__ void __launch_bounds__(256) k_tsdf_slice(float4* __restrict__ out, size_t opitch4, int axis, int v,
                                                    const float2* __restrict__ cv, int W, int H, int D, int ow, int oh) {
    const int a = blockIdx.x * 32 + threadIdx.x, b = blockIdx.y * 8 + threadIdx.y;
    if (a >= ow || b >= oh) return;
    const int x = axis == 0 ? v : a, y = axis == 0 ? a : (axis == 1 ? v : b), z = axis == 2 ? v : b;
    const float t = fminf(fmaxf(cv[((size_t)z * H + y) * W + x].x + 0.5f, 0.0f), 1.0f);
    out[(size_t)b * opitch4 + a] = make_float4(t, t, t, 1.0f);
}

cvtpm_status fail(cvtpm_status s, const std::string& m) {
    pm_set_free_error(m);
    return s;
}

bool finite16(const float* m) {
    for (int i = 0; i < 16; ++i)
        if (!isfinite(m[i])) return false;
    return true;
}

}  // namespace

struct cvtpm_tsdf {
    int device;
    int W, H, D;
    float trunc;
    Mat4 g2w;
    float2* vol;
    unsigned char* bricks;     /* marks of the ray casts, behind the volume; NULL: no room for them */
};

/* The bricks cost a pass over the volume and two launches, and save the
 * evaluations of empty samples: time that grows with the rays times an extent,
 * and with the extent alone where the rays are too few to fill the GPU.  Without
 * and with, ms, a scene with a surface: 640x480 rays 96^3 0.112, 0.111, 256^3
 * 0.264, 0.210, 512^3 0.622, 0.496, 768^3 1.06, 1.03, 1024^3 1.58, 1.95; 320x240
 * rays 256^3 0.152, 0.195, 384^3 0.404, 0.339, 512^3 0.534, 0.508, 768^3 0.88,
 * 1.03, 64x512x512 0.136, 0.101, 512x512x64 0.048, 0.053; 1280x960 rays 48^3
 * 0.187, 0.200; 1920x1080 rays 1024^3 5.3, 2.7.  (Empty volumes gain more; where
 * every voxel has weight, 256^3 with 640x480 rays, 0.50 and 0.70.) */
static bool bricks_pay(int W, int H, int D, int dwidth, int dheight) {
    const double rays = (double)dwidth * dheight, extent = ((double)W + H + D) / 3, voxels = (double)W * H * D;
    return extent >= 64 && rays * extent >= 27e6 && voxels <= 2 * (rays + 100000) * extent;
}

/* bricks of 1 << sh voxels along an extent */
static int tsdf_bricks(int extent, int sh) { return (extent + (1 << sh) - 1) >> sh; }

/* Vision::disparityToDepthmap (cvt/vision/Vision.cpp:147-168): the depth
 * (focallength * baseline) / (disparity * dispscale) where the scaled
 * disparity exceeds dispthres, else 0.  8 bytes per pixel: HBM-bound. */
__global__ void __launch_bounds__(256) k_disparity_to_depth(float* __restrict__ depth, size_t dp,
                                                            const float* __restrict__ disp, size_t sp, int W, int H,
                                                            float dispscale, float fb, float thres) {
    const int x = blockIdx.x * 64 + threadIdx.x, y = blockIdx.y * 4 + threadIdx.y;
    if (x >= W || y >= H) return;
    const float d = disp[(size_t)y * sp + x] * dispscale;
    depth[(size_t)y * dp + x] = d > thres ? fb / d : 0.0f;
}

extern "C" {

cvtpm_status cvtpm_tsdf_projection(const float* intrinsics, const float* extrinsics, float* proj) {
    if (!intrinsics || !extrinsics || !proj) return fail(CVTPM_ERR_INVALID_ARGUMENT, "tsdf projection: NULL argument");
    Mat4 K = {{intrinsics[0], intrinsics[1], intrinsics[2], 0.0f, intrinsics[3], intrinsics[4], intrinsics[5], 0.0f,
               intrinsics[6], intrinsics[7], intrinsics[8], 0.0f, 0.0f, 0.0f, 0.0f, 1.0f}};   /* Matrix3::toMatrix4 */
    Mat4 E;
    memcpy(E.m, extrinsics, sizeof E.m);
    const Mat4 P = mat4_mul(K, E);   /* proj = K.toMatrix4(); proj *= extrinsics (TSDFVolume.cpp:79-84) */
    memcpy(proj, P.m, sizeof P.m);
    return CVTPM_OK;
}

cvtpm_status cvtpm_tsdf_create(cvtpm_tsdf** out, int device, const float* grid_to_world, int width, int height,
                               int depth, float truncation) {
    if (!out || !grid_to_world) return fail(CVTPM_ERR_INVALID_ARGUMENT, "tsdf create: NULL argument");
    *out = nullptr;
    if (width < 2 || height < 2 || depth < 2 || width > 4096 || height > 4096 || depth > 4096)
        return fail(CVTPM_ERR_SIZE, "tsdf create: each dimension must be 2..4096");
    if (!finite16(grid_to_world) || !(truncation > 0.0f)) return fail(CVTPM_ERR_INVALID_ARGUMENT, "tsdf create: bad grid-to-world or truncation");
    if (cudaSetDevice(device) != cudaSuccess) return fail(CVTPM_ERR_CUDA, "tsdf create: cudaSetDevice");
    cvtpm_tsdf* v = new cvtpm_tsdf();
    v->device = device;
    v->W = width; v->H = height; v->D = depth;
    v->trunc = truncation;
    memcpy(v->g2w.m, grid_to_world, sizeof v->g2w.m);
    const size_t bytes = sizeof(float2) * (size_t)width * height * depth;
    size_t bricks = 0;
    for (int sh : {TSDF_FINE, TSDF_COARSE})
        bricks += (size_t)tsdf_bricks(width, sh) * tsdf_bricks(height, sh) * tsdf_bricks(depth, sh);
    if (cudaMalloc(&v->vol, bytes + bricks) == cudaSuccess) {
        v->bricks = (unsigned char*)v->vol + bytes;
    } else if (cudaGetLastError(), cudaMalloc(&v->vol, bytes) != cudaSuccess) {
        cudaGetLastError();
        delete v;
        return fail(CVTPM_ERR_ALLOC, "tsdf create: volume allocation failed");
    }
    *out = v;
    return CVTPM_OK;
}

cvtpm_status cvtpm_tsdf_destroy(cvtpm_tsdf* v) {
    if (!v) return CVTPM_ERR_INVALID_ARGUMENT;
    cudaSetDevice(v->device);
    cudaFree(v->vol);
    delete v;
    return CVTPM_OK;
}

cvtpm_status cvtpm_tsdf_info(const cvtpm_tsdf* v, int* width, int* height, int* depth, void** data) {
    if (!v) return fail(CVTPM_ERR_INVALID_ARGUMENT, "tsdf info: NULL volume");
    if (width) *width = v->W;
    if (height) *height = v->H;
    if (depth) *depth = v->D;
    if (data) *data = v->vol;
    return CVTPM_OK;
}

cvtpm_status cvtpm_tsdf_clear(cvtpm_tsdf* v, float weight, void* stream) {
    if (!v) return fail(CVTPM_ERR_INVALID_ARGUMENT, "tsdf clear: NULL volume");
    cudaSetDevice(v->device);
    if (TSDF_CLEAR_VEC) {
        const size_t n = (size_t)v->W * v->H * v->D, th = (n + 1) / 2;
        k_tsdf_clear_vec<<<(unsigned)((th + 255) / 256), 256, 0, (cudaStream_t)stream>>>((float4*)v->vol, n, weight);
    } else {
        k_tsdf_clear<<<dim3((v->W + 31) / 32, (v->H + 7) / 8, v->D), dim3(32, 8), 0, (cudaStream_t)stream>>>(
            v->vol, v->W, v->H, v->D, weight);
    }
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? CVTPM_OK : fail(CVTPM_ERR_CUDA, std::string("tsdf clear: ") + cudaGetErrorString(e));
}

cvtpm_status cvtpm_tsdf_add_depthmap(cvtpm_tsdf* v, const float* proj, const float* depthmap, int dwidth, int dheight,
                                     size_t dpitch, float scale, void* stream) {
    if (!v || !proj || !depthmap) return fail(CVTPM_ERR_INVALID_ARGUMENT, "tsdf add: NULL argument");
    if (dwidth < 1 || dheight < 1) return fail(CVTPM_ERR_SIZE, "tsdf add: empty depth map");
    if (dpitch % 4 || dpitch < (size_t)dwidth * 4) return fail(CVTPM_ERR_INVALID_ARGUMENT, "tsdf add: bad depth map pitch");
    if (!finite16(proj)) return fail(CVTPM_ERR_INVALID_ARGUMENT, "tsdf add: non-finite projection");
    Mat4 P;
    memcpy(P.m, proj, sizeof P.m);
    const DMat4 T = to_dev(mat4_mul(P, v->g2w));   /* projall = proj * g2w (TSDFVolume.cpp:64) */
    cudaSetDevice(v->device);
    k_tsdf_add<<<dim3((v->W + 31) / 32, (v->H + 7) / 8, (v->D + TSDF_ZPT - 1) / TSDF_ZPT), dim3(32, 8), 0,
                 (cudaStream_t)stream>>>(
        v->vol, v->W, v->H, v->D, depthmap, dpitch / 4, dwidth, dheight, scale, T, v->trunc);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? CVTPM_OK : fail(CVTPM_ERR_CUDA, std::string("tsdf add: ") + cudaGetErrorString(e));
}

int cvtpm_tool_tsdf_bricks(int width, int height, int depth, int dwidth, int dheight) {
    return bricks_pay(width, height, depth, dwidth, dheight) ? 1 : 0;
}

cvtpm_status cvtpm_tsdf_raycast(cvtpm_tsdf* v, const float* proj, float* depthmap, int dwidth, int dheight,
                                size_t dpitch, float scale, void* stream) {
    if (!v || !proj || !depthmap) return fail(CVTPM_ERR_INVALID_ARGUMENT, "tsdf raycast: NULL argument");
    if (dwidth < 1 || dheight < 1) return fail(CVTPM_ERR_SIZE, "tsdf raycast: empty depth map");
    if (dpitch % 4 || dpitch < (size_t)dwidth * 4) return fail(CVTPM_ERR_INVALID_ARGUMENT, "tsdf raycast: bad depth map pitch");
    if (!finite16(proj)) return fail(CVTPM_ERR_INVALID_ARGUMENT, "tsdf raycast: non-finite projection");
    Mat4 P;
    memcpy(P.m, proj, sizeof P.m);
    const Mat4 all = mat4_mul(P, v->g2w);
    const DMat4 T = to_dev(all), Ti = to_dev(mat4_inverse(all));
    const int max_steps = 2 * (v->W > v->H ? (v->W > v->D ? v->W : v->D) : (v->H > v->D ? v->H : v->D)) + 16;
    cudaSetDevice(v->device);
    BrickGrid g = {nullptr, nullptr, tsdf_bricks(v->W, TSDF_FINE), tsdf_bricks(v->H, TSDF_FINE),
                   tsdf_bricks(v->W, TSDF_COARSE), tsdf_bricks(v->H, TSDF_COARSE)};
    if (v->bricks && bricks_pay(v->W, v->H, v->D, dwidth, dheight)) {
        /* formed anew for each cast: the caller may write the volume (cvtpm_tsdf_info) */
        const int fd = tsdf_bricks(v->D, TSDF_FINE), cd = tsdf_bricks(v->D, TSDF_COARSE);
        unsigned char *fine = v->bricks, *coarse = fine + (size_t)g.fw * g.fh * fd;
        const int threads = v->W < 256 ? (v->W + 31) / 32 * 32 : 256;
        k_tsdf_bricks<<<dim3((v->W + threads - 1) / threads, g.fh, fd), threads, 0, (cudaStream_t)stream>>>(v->vol, v->W, v->H, v->D, fine, g);
        k_tsdf_coarse<<<(g.cw * g.ch * cd + 7) / 8, 256, 0, (cudaStream_t)stream>>>(fine, coarse, g, fd, cd);
        g.fine = fine;
        g.coarse = coarse;
    }
    (g.fine ? k_tsdf_raycast<true> : k_tsdf_raycast<false>)<<<dim3((dwidth + 31) / 32, (dheight + 7) / 8), dim3(32, 8), 0, (cudaStream_t)stream>>>(
        depthmap, dpitch / 4, dwidth, dheight, v->vol, v->W, v->H, v->D, g, Ti, T, scale, max_steps);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? CVTPM_OK : fail(CVTPM_ERR_CUDA, std::string("tsdf raycast: ") + cudaGetErrorString(e));
}

cvtpm_status cvtpm_tsdf_slice(cvtpm_tsdf* v, int axis, int index, float* rgba, size_t pitch, void* stream) {
    if (!v || !rgba) return fail(CVTPM_ERR_INVALID_ARGUMENT, "tsdf slice: NULL argument");
    if (axis < 0 || axis > 2) return fail(CVTPM_ERR_INVALID_ARGUMENT, "tsdf slice: axis must be 0 (x), 1 (y) or 2 (z)");
    const int ext = axis == 0 ? v->W : (axis == 1 ? v->H : v->D);
    if (index < 0 || index >= ext) return fail(CVTPM_ERR_SIZE, "tsdf slice: index outside the volume");
    const int ow = axis == 0 ? v->H : v->W, oh = axis == 2 ? v->H : v->D;
    if (pitch % 16 || pitch < (size_t)ow * 16) return fail(CVTPM_ERR_INVALID_ARGUMENT, "tsdf slice: bad pitch");
    cudaSetDevice(v->device);
    k_tsdf_slice<<<dim3((ow + 31) / 32, (oh + 7) / 8), dim3(32, 8), 0, (cudaStream_t)stream>>>(
        (float4*)rgba, pitch / 16, axis, index, v->vol, v->W, v->H, v->D, ow, oh);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? CVTPM_OK : fail(CVTPM_ERR_CUDA, std::string("tsdf slice: ") + cudaGetErrorString(e));
}

cvtpm_status cvtpm_tsdf_save_raw(cvtpm_tsdf* v, const char* path, int weighted) {
    if (!v || !path) return fail(CVTPM_ERR_INVALID_ARGUMENT, "tsdf save: NULL argument");
    const size_t n = (size_t)v->W * v->H * v->D;
    std::vector<float> host(2 * n);
    cudaSetDevice(v->device);
    if (cudaMemcpy(host.data(), v->vol, sizeof(float) * 2 * n, cudaMemcpyDeviceToHost) != cudaSuccess)
        return fail(CVTPM_ERR_CUDA, "tsdf save: copy failed");
    FILE* f = fopen(path, "wb");
    if (!f) return fail(CVTPM_ERR_IO, std::string("tsdf save: cannot open ") + path);
    bool ok;
    if (weighted) {   /* (tsdf, weight) pairs; else the tsdf values alone (TSDFVolume.cpp:130-152) */
        ok = fwrite(host.data(), sizeof(float), 2 * n, f) == 2 * n;
    } else {
        for (size_t i = 0; i < n; ++i) host[i] = host[2 * i];
        ok = fwrite(host.data(), sizeof(float), n, f) == n;
    }
    ok = (fclose(f) == 0) && ok;
    return ok ? CVTPM_OK : fail(CVTPM_ERR_IO, std::string("tsdf save: write failed for ") + path);
}

}  // extern "C"

extern "C" cvtpm_status cvtpm_disparity_to_depth(float* depth, size_t depth_pitch, const float* disparity,
                                                 size_t disp_pitch, int width, int height, float dispscale,
                                                 float focallength, float baseline, float dispthres, void* stream) {
    if (!depth || !disparity) return fail(CVTPM_ERR_INVALID_ARGUMENT, "disparity to depth: NULL argument");
    if (width < 1 || height < 1) return fail(CVTPM_ERR_SIZE, "disparity to depth: empty image");
    if (depth_pitch % 4 || disp_pitch % 4 || depth_pitch < (size_t)width * 4 || disp_pitch < (size_t)width * 4)
        return fail(CVTPM_ERR_INVALID_ARGUMENT, "disparity to depth: bad pitch");
    const float fb = focallength * baseline;   /* Vision.cpp:153, in float */
    k_disparity_to_depth<<<dim3((width + 63) / 64, (height + 3) / 4), dim3(64, 4), 0, (cudaStream_t)stream>>>(
        depth, depth_pitch / 4, disparity, disp_pitch / 4, width, height, dispscale, fb, dispthres);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? CVTPM_OK : fail(CVTPM_ERR_CUDA, std::string("disparity to depth: ") + cudaGetErrorString(e));
}
