// compat.cu -- COMPAT arithmetic: the reference's FP32 Siddon traversal,
// reproduced operation for operation, with one thread per ray and the whole
// traversal in registers.
//
// The reference runs every traversal step as separate launches over all rays
// (siddon_sort_alpha, siddon_fp_calc_ray_path / siddon_bp_calc_ray_path,
// siddon_add, the atomic scatter kernel and a full-volume siddon_add_bp per
// step; CT_Recon/hf_siddon_class.hpp:195-225, 313-347), with a blocking
// device-to-host copy per view to find the step count.  Here each thread
// carries one ray from set-up to its end segment: no per-step launches, no
// memsets, no host synchronisation.  The per-ray arithmetic is the
// reference's own: every expression below keeps the operand order of the
// reference line it restates, so that the compiler forms the same FMAs and
// the intrinsics (__fdividef, __fdiv_rz, cospif, sinpif, __float2int_rz) see
// the same operands.  Float-to-unsigned conversions of run-time values
// (float plane indices passed as unsigned) are made explicit with the
// saturating device conversion (NaN -> 0), which is what the hardware does.
// The reference also stores the constant CUDART_NAN_F into its unsigned
// ray mask (calc_mask, the parallel-axis branch of siddon_calc_indices,
// bound_index).  Converting NaN to an integer is undefined behaviour in C++,
// and nvcc's optimizer drops those stores: the reference's sm_100a build
// keeps mask = 1 for every ray (measured on all test geometries, misses and
// axis-parallel rays included).  COMPAT reproduces the GPU build, so the mask
// is never cleared here either.
//
// Back projection keeps the reference's ray-driven scatter, but accumulates the
// contributions len*img of the views of a call, as many as are of like magnitude, in
// 64-bit fixed point (integer atomics, exact and order independent) and rounds once to
// float, so the result is deterministic; the reference sums with float atomics in
// arbitrary order.
#include "internal.h"

#include <cooperative_groups.h>

#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>

namespace rb {
namespace compat {

#define RB_CUDART_NAN_F __int_as_float(0x7FFFFFFF)

struct Ray {
    float p1[3], p2[3];
    float d12, amin, amax;
    unsigned mask;
    float ai[3], af[3], da[3];
    unsigned dindex;
};

// pixel_iterate2 (hf_cuda_kernels.cuh:92-97)
__device__ __forceinline__ float pixel_center(float NumPixels, float PixelsDimMm, float Mag, int iterator)
{
    float result = __fdividef(-(NumPixels - 1.0f), 2.0f) * PixelsDimMm * Mag +
                   __fdividef((float)iterator, NumPixels) * NumPixels * PixelsDimMm * Mag;
    return __fdiv_rz(rintf(result * 100000.0f), 100000.0f);
}

// find_index (siddon_device_kernelsMLEM.cuh:151-185)
__device__ __forceinline__ float plane_index(float index, float amin, float amax, float p1, float p2,
                                             float plane1, float dplane)
{
    if (index > 0.0f) {
        float low = floorf(index), high = ceilf(index);
        float plane_low = (plane1 + dplane * (low - 1.0f));
        float plane_high = (plane1 + dplane * (high - 1.0f));
        float alow = __fdividef(plane_low - p1, p2 - p1);
        float ahigh = __fdividef(plane_high - p1, p2 - p1);
        if (alow >= amin && alow <= amax) return low;
        else if (ahigh >= amin && ahigh <= amax) return high;
        else return RB_CUDART_NAN_F;
    }
    return RB_CUDART_NAN_F;
}

// alpha_float (siddon_device_kernelsMLEM.cuh:218-237); mn, mx arrive unsigned
__device__ __forceinline__ float plane_alpha(unsigned mn, unsigned mx, float p1, float p2, float plane1,
                                            float dplane)
{
    float plane;
    if ((p2 - p1) > 0 && (mx - mn) > 0) {
        plane = plane1 + dplane * ((float)mn - 1.0f);
        return __fdividef(plane - p1, p2 - p1);
    } else if ((p2 - p1) < 0 && (mx - mn) > 0) {
        plane = plane1 + dplane * ((float)mx - 1.0f);
        return __fdividef(plane - p1, p2 - p1);
    }
    return RB_CUDART_NAN_F;
}

// siddon_calc_indices (siddon_device_kernelsMLEM.cuh:240-270) with bound_index (:50-58)
__device__ __forceinline__ unsigned axis_indices(float& ai, float& af, unsigned& mask, float p1, float p2,
                                                 float plane1, float plane2, float Nplanes, float amin,
                                                 float amax, float dplane)
{
    float ix, iy;
    if ((p2 - p1) > 0) {
        ix = Nplanes - __fdividef((plane2 - amin * (p2 - p1) - p1), dplane);
        iy = 1.0f + __fdividef((p1 + amax * (p2 - p1) - plane1), dplane);
    } else if ((p2 - p1) < 0) {
        ix = Nplanes - __fdividef((plane2 - amax * (p2 - p1) - p1), dplane);
        iy = 1.0f + __fdividef((p1 + amin * (p2 - p1) - plane1), dplane);
    } else {
        ix = 0;
        iy = 0;  // (the reference's mask store here is dropped by nvcc)
    }
    ix = (float)mask * plane_index(ix, amin, amax, p1, p2, plane1, dplane);
    iy = (float)mask * plane_index(iy, amin, amax, p1, p2, plane1, dplane);
    if ((iy - ix) < 0 && ix <= 1 && iy <= 1) {
        ix = 0;
        iy = 0;  // bound_index; its mask store is dropped likewise
    }
    ai = (float)mask * plane_alpha(__float2uint_rz(ix), __float2uint_rz(iy), p1, p2, plane1, dplane);
    af = (float)mask * plane_alpha(__float2uint_rz(iy), __float2uint_rz(ix), p1, p2, plane1, dplane);
    return __float2uint_rz(iy - ix);
}

// calc_points12 (siddon_device_kernelsMLEM.cuh:305-331) + siddon_alpha_limits
// (siddon_kernelsMLEM.cuh:103-149)
__device__ __forceinline__ void setup(const CompatGeom& G, float angle, int u, int v, Ray& r)
{
    float det_x = pixel_center(G.NumAxPixels_f, G.AxPixDimMm, G.M, u);
    float det_y = G.R - G.Rf;
    float det_z = pixel_center(G.NumTAxPixels_f, G.TAxPixDimMm, G.M, v);
    det_x = __fdividef(G.R, (G.Ry + G.RM[3] * det_x + G.RM[5] * det_z)) * (G.RM[0] * det_x + G.RM[2] * det_z + G.Dx);
    det_z = __fdividef(G.R, (G.Ry + G.RM[3] * det_x + G.RM[5] * det_z)) * (G.RM[6] * det_x + G.RM[8] * det_z + G.Dz);
    float cos_a = cospif(__fdividef(angle, 180.0f));
    float sin_a = sinpif(__fdividef(angle, 180.0f));
    r.p1[0] = G.Xs[0] * cos_a + G.Xs[1] * sin_a;
    r.p1[1] = -G.Xs[0] * sin_a + G.Xs[1] * cos_a;
    r.p1[2] = G.Xs[2];
    r.p2[0] = det_x * cos_a + det_y * sin_a;
    r.p2[1] = -det_x * sin_a + det_y * cos_a;
    r.p2[2] = det_z;
    r.d12 = sqrtf((r.p2[0] - r.p1[0]) * (r.p2[0] - r.p1[0]) + (r.p2[1] - r.p1[1]) * (r.p2[1] - r.p1[1]) +
                  (r.p2[2] - r.p1[2]) * (r.p2[2] - r.p1[2]));
    float a1[3], aN[3];
    for (int k = 0; k < 3; ++k) {  // calc_alpha_1N (siddon_device_kernelsMLEM.cuh:71-85)
        if ((r.p2[k] - r.p1[k]) != 0) {
            a1[k] = __fdividef(G.Pi[k] - r.p1[k], r.p2[k] - r.p1[k]);
            aN[k] = __fdividef(G.Pf[k] - r.p1[k], r.p2[k] - r.p1[k]);
        } else {
            a1[k] = RB_CUDART_NAN_F;
            aN[k] = RB_CUDART_NAN_F;
        }
    }
    float amin = fmaxf(fmaxf(fmaxf(0, fminf(a1[0], aN[0])), fminf(a1[1], aN[1])), fminf(a1[2], aN[2]));
    float amax = fminf(fminf(fminf(1, fmaxf(a1[0], aN[0])), fmaxf(a1[1], aN[1])), fmaxf(a1[2], aN[2]));
    unsigned mask = 1u;  // calc_mask (:88-98) as the GPU build evaluates it
    amin = (float)mask * amin;
    amax = (float)mask * amax;
    unsigned idx[3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
        idx[k] = axis_indices(r.ai[k], r.af[k], mask, r.p1[k], r.p2[k], G.Pi[k], G.Pf[k], (float)G.dims[k] + 1.0f,
                              amin, amax, G.Pd[k]);
    r.dindex = idx[0] + 1 + idx[1] + 1 + idx[2] + 1 + 1;
#pragma unroll
    for (int k = 0; k < 3; ++k) r.da[k] = fabsf(__fdividef(G.Pd[k], r.p2[k] - r.p1[k]));  // delta_alpha (:100-113)
    r.mask = mask;
    r.amin = amin;
    r.amax = amax;
}

// alpha_bound (siddon_device_kernelsMLEM.cuh:134-148)
__device__ __forceinline__ float clamp_alpha(float a, float ai, float af, float amax)
{
    if (a >= ai && a <= af) return a;
    else if (a > af) return amax;
    return RB_CUDART_NAN_F;
}

__device__ __forceinline__ bool same_bits(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }

struct State {
    float a[3];
    float cur, next;
};

// siddon_begin (siddon_kernelsMLEM.cuh:283-303)
__device__ __forceinline__ void begin(const Ray& r, State& s)
{
    s.a[0] = r.mask * r.ai[0];
    s.a[1] = r.mask * r.ai[1];
    s.a[2] = r.mask * r.ai[2];
    s.next = fminf(fminf(r.ai[0], r.ai[1]), r.ai[2]);
    s.cur = RB_CUDART_NAN_F;
}

// siddon_sort_alpha (siddon_kernelsMLEM.cuh:153-190).  Returns true when the
// step left the state unchanged with next == current: every later step
// repeats it and yields a zero-length segment, so the caller may stop.
__device__ __forceinline__ bool step(const Ray& r, State& s)
{
    const float a0 = s.a[0], a1 = s.a[1], a2 = s.a[2], n0 = s.next;
    s.cur = s.next;
    if (s.cur == s.a[0]) {
        s.a[0] = s.a[0] + r.da[0];
        s.a[0] = clamp_alpha(s.a[0], r.ai[0], r.af[0], r.amax);
    } else if (s.cur == s.a[1]) {
        s.a[1] = s.a[1] + r.da[1];
        s.a[1] = clamp_alpha(s.a[1], r.ai[1], r.af[1], r.amax);
    } else if (s.cur == s.a[2]) {
        s.a[2] = s.a[2] + r.da[2];
        s.a[2] = clamp_alpha(s.a[2], r.ai[2], r.af[2], r.amax);
    }
    s.next = fminf(fminf(s.a[0], s.a[1]), s.a[2]);
    return same_bits(a0, s.a[0]) && same_bits(a1, s.a[1]) && same_bits(a2, s.a[2]) && same_bits(n0, s.next) &&
           same_bits(s.next, s.cur);
}

// Segment of siddon_fp_calc_ray_path / siddon_bp_calc_ray_path /
// siddon_fp_end / siddon_bp_end (siddon_kernelsMLEM.cuh:193-279, 307-411):
// midpoint voxel and length; -1 when there is no in-range segment.
__device__ __forceinline__ int segment(const CompatGeom& G, const Ray& r, float a_hi, float a_lo, float& len)
{
    int ix = -1, iy = -1, iz = -1;
    float ray_length = 0.0f;
    if (a_hi > a_lo) {
        float alpha_mid = __fdividef((a_hi + a_lo), 2.0f);
        ray_length = r.d12 * (a_hi - a_lo);
        ix = __float2int_rz((__fdividef((r.p1[0] + alpha_mid * (r.p2[0] - r.p1[0]) - G.Pi[0]), G.Pd[0])));
        iy = __float2int_rz((__fdividef((r.p1[1] + alpha_mid * (r.p2[1] - r.p1[1]) - G.Pi[1]), G.Pd[1])));
        iz = __float2int_rz((__fdividef((r.p1[2] + alpha_mid * (r.p2[2] - r.p1[2]) - G.Pi[2]), G.Pd[2])));
    }
    len = ray_length;
    if (ix >= 0 && ix < G.dims[0] && iy >= 0 && iy < G.dims[1] && iz >= 0 && iz < G.dims[2])
        return (int)((unsigned)iz * (unsigned)(G.dims[1] * G.dims[0]) + (unsigned)iy * (unsigned)G.dims[0] + (unsigned)ix);
    return -1;
}

// Offsets of a voxel's neighbours along each axis in the image a projector reads or adds
// to: {1, X, X Y} for the caller's layout, {Z, X Z, 1} where z runs fastest.
struct VoxelStrides {
    int x, y, z;
};

// ---- kernels -------------------------------------------------------------------

__device__ __forceinline__ float view_angle(const float* angles, unsigned view) { return angles[view]; }

// Per-view loopN = max delta_index (siddon_commons::a_calc_initial_limits,
// hf_siddon_class.hpp:93-106), computed on the device.
__global__ void loopn_kernel(CompatGeom G, const float* __restrict__ angles, unsigned view0,
                             unsigned* __restrict__ loopN)
{
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    const int v = blockIdx.y * blockDim.y + threadIdx.y;
    const unsigned view = view0 + blockIdx.z;
    unsigned d = 0;
    if (u < G.Nu && v < G.Nv) {
        Ray r;
        setup(G, view_angle(angles, view), u, v, r);
        d = r.dindex;
    }
    for (int o = 16; o > 0; o >>= 1) d = max(d, __shfl_xor_sync(0xffffffffu, d, o));
    if ((threadIdx.x & 31) == 0 && d) atomicMax(&loopN[view], d);
}

__global__ void setup_dump_kernel(CompatGeom G, float angle, float* amin, float* amax, float* d12, unsigned* mask,
                                  float* ai, float* af, float* da, float* p1, float* p2, unsigned* dindex)
{
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    const int v = blockIdx.y * blockDim.y + threadIdx.y;
    if (u >= G.Nu || v >= G.Nv) return;
    const size_t n = (size_t)u + (size_t)v * G.Nu;
    Ray r;
    setup(G, angle, u, v, r);
    amin[n] = r.amin;
    amax[n] = r.amax;
    d12[n] = r.d12;
    mask[n] = r.mask;
    dindex[n] = r.dindex;
    for (int k = 0; k < 3; ++k) {
        ai[3 * n + k] = r.ai[k];
        af[3 * n + k] = r.af[k];
        da[3 * n + k] = r.da[k];
        p1[3 * n + k] = r.p1[k];
        p2[3 * n + k] = r.p2[k];
    }
}

__global__ void trace_kernel(CompatGeom G, float angle, unsigned loopN, int nrays, const int* __restrict__ rays,
                             int cap, int* __restrict__ idx_out, float* __restrict__ len_out)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= nrays) return;
    const int n = rays[q];
    Ray r;
    setup(G, angle, n % G.Nu, n / G.Nu, r);
    State s;
    begin(r, s);
    int* io = idx_out + (size_t)q * cap;
    float* lo = len_out + (size_t)q * cap;
    for (int k = 0; k < cap; ++k) {
        io[k] = -1;
        lo[k] = 0.0f;
    }
    unsigned k = 0;
    bool fixed = false;
    for (; k < loopN && !fixed; ++k) {
        fixed = step(r, s);
        float len;
        int id = segment(G, r, s.next, s.cur, len);
        if ((int)k < cap) {
            io[k] = id;
            lo[k] = id >= 0 ? len : 0.0f;
        }
    }
    float len;
    int id = segment(G, r, r.amax, s.cur, len);
    if ((int)loopN < cap) {
        io[loopN] = id;
        lo[loopN] = id >= 0 ? len : 0.0f;
    }
}

// The traversal of one ray as the projectors run it: step() and segment() above with
// the axis selected instead of branched on (three quarters of the work is shared
// by the axes), the fixed point looked for every eighth step -- every step past it
// repeats it with a segment of length zero -- and, with POW2, the divisions by
// power-of-two voxel sizes as exact products.  emit(in, voxel, length) is called for
// every step in order, and for the end segment; in: there is a segment, in a voxel of
// the volume.
template <bool POW2, class Emit>
__device__ __forceinline__ void walk(const CompatGeom& G, const Ray& r, unsigned L, VoxelStrides V, Emit emit)
{
    const float dx = r.p2[0] - r.p1[0], dy = r.p2[1] - r.p1[1], dz = r.p2[2] - r.p1[2];
    float a0 = r.mask * r.ai[0], a1 = r.mask * r.ai[1], a2 = r.mask * r.ai[2];  // begin()
    float next = fminf(fminf(r.ai[0], r.ai[1]), r.ai[2]), cur = RB_CUDART_NAN_F;
    auto part = [&](float hi, float lo) {  // segment()
        const float mid = __fdividef((hi + lo), 2.0f);
        const float len = r.d12 * (hi - lo);
        const float fx = r.p1[0] + mid * dx - G.Pi[0], fy = r.p1[1] + mid * dy - G.Pi[1], fz = r.p1[2] + mid * dz - G.Pi[2];
        const int ix = __float2int_rz(POW2 ? fx * G.inv_Pd[0] : __fdividef(fx, G.Pd[0]));
        const int iy = __float2int_rz(POW2 ? fy * G.inv_Pd[1] : __fdividef(fy, G.Pd[1]));
        const int iz = __float2int_rz(POW2 ? fz * G.inv_Pd[2] : __fdividef(fz, G.Pd[2]));
        const bool in = hi > lo && (unsigned)ix < (unsigned)G.dims[0] && (unsigned)iy < (unsigned)G.dims[1] &&
                        (unsigned)iz < (unsigned)G.dims[2];
        emit(in, ix * V.x + iy * V.y + iz * V.z, len);
    };
    // a ray with no plane to start from (most that miss the volume): NaN throughout, and
    // no step gives a segment
    if (next != next) return;
    auto advance = [&] {  // siddon_sort_alpha, as step() has it
        cur = next;
        const bool bx = cur == a0, by = !bx && cur == a1, bz = !bx && !by && cur == a2;
        const float da = bx ? r.da[0] : by ? r.da[1] : r.da[2];
        const float ai = bx ? r.ai[0] : by ? r.ai[1] : r.ai[2];
        const float af = bx ? r.af[0] : by ? r.af[1] : r.af[2];
        const float n = clamp_alpha(cur + da, ai, af, r.amax);
        a0 = bx ? n : a0;
        a1 = by ? n : a1;
        a2 = bz ? n : a2;
        next = fminf(fminf(a0, a1), a2);
        part(next, cur);
    };
    unsigned k = 0;
    bool fixed = false;
    for (; k + 8 <= L && !fixed; k += 8) {
#pragma unroll
        for (int q = 0; q < 7; ++q) advance();
        const float b0 = a0, b1 = a1, b2 = a2, bn = next;
        advance();
        fixed = same_bits(b0, a0) && same_bits(b1, a1) && same_bits(b2, a2) && same_bits(bn, next) && same_bits(next, cur);
    }
    if (!fixed)
        for (; k < L; ++k) advance();
    part(r.amax, cur);
}

// Bound by instruction issue (83 % of peak).  256^3 / 360 views / 512^2: forward 19.2 ->
// 13.5 ms and scatter 19.4 -> 14.1 ms, from lanes along detector columns that branched
// apart at every step, in a grid that had every view's rays cross an accumulator larger
// than L2 (41 GB of DRAM traffic per scatter, now 0.8 GB).
// Rays of a CTA: 32 detector rows (lanes) x 8 detector columns.  The rays of one
// detector column cross nearly the same (x, y) voxel columns, so a warp's lanes step
// alike, and their voxels lie next to each other in an image whose z runs fastest.
// Grid {columns / 8, views, rows / 32}: the views of one row group are in flight
// together, whose rays meet a slab of slices.
constexpr int kRayRows = 32, kRayCols = 8;

// Forward projection: image = sum over steps, in step order, of len*f[idx],
// each product and each sum rounded once (siddon_fp_calc_ray_path writes the
// product, siddon_add adds it).  mode 0: store Hf; mode 1: store
// divide1(g, Hf) (hf_cuda_kernels.cuh:370-387) and track max |ratio| per view.
template <int MODE, bool POW2>
__global__ void __launch_bounds__(kRayRows * kRayCols, 4) fp_kernel(CompatGeom G, const float* __restrict__ angles,
                                                                 const unsigned* __restrict__ loopN, unsigned view0,
                                                                 VoxelStrides V, const float* __restrict__ vol,
                                                                 const float* __restrict__ g, float* __restrict__ out,
                                                                 unsigned* __restrict__ maxabs)
{
    __shared__ float tile[kRayCols][kRayRows + 1];
    const int u0 = blockIdx.x * kRayCols, v0 = blockIdx.z * kRayRows;
    const unsigned view = view0 + blockIdx.y;
    {
        const int u = u0 + threadIdx.y, v = v0 + threadIdx.x;
        float acc = 0.0f;
        if (u < G.Nu && v < G.Nv) {
            Ray r;
            setup(G, view_angle(angles, view), u, v, r);
            // Rays with mask 0 are not skipped: when a later axis clears the mask the
            // traversal can still produce segments, exactly as in the reference.
            walk<POW2>(G, r, loopN[view], V, [&](bool in, int id, float len) {
                const float t = in ? __fmul_rn(len, __ldg(vol + id)) : 0.0f;
                acc = __fadd_rn(acc, t);
            });
        }
        tile[threadIdx.y][threadIdx.x] = acc;
    }
    __syncthreads();
    // written eight columns (one 32-byte sector) at a time
    const int t = threadIdx.y * kRayRows + threadIdx.x;
    const int u = u0 + t % kRayCols, v = v0 + t / kRayCols;
    const bool in = u < G.Nu && v < G.Nv;
    const size_t n = (size_t)blockIdx.y * G.Nu * G.Nv + (size_t)u + (size_t)v * G.Nu;
    const float acc = tile[t % kRayCols][t / kRayCols];
    if (MODE == 0) {
        if (in) out[n] = acc;
    } else {
        float ratio = 0.0f;
        if (in) {
            ratio = (acc != 0) ? __fdividef(g[n], acc) : 0.0f;
            out[n] = ratio;
        }
        // one atomic per warp, where it raises the view's maximum: every ray of the
        // block belongs to this view, and a max does not depend on the order it is taken in
        const unsigned bits = __reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(ratio)));
        if (threadIdx.x == 0 && bits > *(volatile unsigned*)(maxabs + view)) atomicMax(&maxabs[view], bits);
    }
}

__global__ void maxabs_kernel(const float* __restrict__ img, size_t n, unsigned* __restrict__ out)
{
    unsigned m = 0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        m = max(m, __float_as_uint(fabsf(img[i])));
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m) atomicMax(out, m);
}

// Fixed-point scale for a view.  Every segment lies on its ray, so
// |len*img| <= maxabs * max_len with max_len >= every source-detector
// distance; a voxel receives at most 2^count_bits contributions (one per ray
// of the view), so with scale = 2^F, F = 62 - count_bits - e and
// maxabs*max_len < 2^e, the per-voxel sum stays below 2^62.  INT_MIN where there is
// nothing to add (all zero), or a value is not finite.
__device__ __forceinline__ int fix_exponent(unsigned maxabs_bits, float max_len, int count_bits)
{
    const float m = __uint_as_float(maxabs_bits);
    if (!(m > 0.0f) || !isfinite(m)) return INT_MIN;
    int e;
    frexp((double)m * (double)max_len, &e);
    return min(62 - count_bits - e, 200);
}

__device__ __forceinline__ double fix_scale(unsigned maxabs_bits, float max_len, int count_bits)
{
    const int F = fix_exponent(maxabs_bits, max_len, count_bits);
    return F == INT_MIN ? 0.0 : ldexp(1.0, F);
}

// The views of one call that share an accumulator.  A band is every view whose own
// accumulator (bounds len, bits: one view) would have had a quantum no finer than the
// band's (len_all, bits_all: every view of the call, scaled by a magnitude `top` that
// none of them exceeds), so that no contribution is rounded more coarsely for the company
// it keeps.  Views that hold a value that is not finite are in no band, nor are zero ones.
struct BandRule {
    float len, len_all;
    int bits, bits_all;
};

__device__ __forceinline__ bool in_band(unsigned maxabs_bits, unsigned top, const BandRule& R)
{
    if (maxabs_bits > top || top == 0u) return false;
    const int F = fix_exponent(maxabs_bits, R.len, R.bits);
    return F != INT_MIN && F <= fix_exponent(top, R.len_all, R.bits_all);
}

// The largest finite magnitude among the n views of maxabs that come after the band of
// `prev`, or 0 where none is left.  Called by all 256 threads of a block.
__device__ __forceinline__ unsigned next_band(const unsigned* maxabs, unsigned n, unsigned prev, const BandRule& R)
{
    __shared__ unsigned best;
    const unsigned t = threadIdx.y * blockDim.x + threadIdx.x;
    __syncthreads();
    if (t == 0) best = 0u;
    __syncthreads();
    unsigned m = 0u;
    for (unsigned i = t; i < n; i += 256u) {
        const unsigned b = maxabs[i];
        if (b < prev && !in_band(b, prev, R)) m = max(m, b);
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if ((t & 31u) == 0u && m) atomicMax(&best, m);
    __syncthreads();
    return best;
}

// Back projection scatter of a block's rays (detector columns u0 .., rows v0 ..): per
// in-range segment, len*img[n] added in 64-bit fixed point (siddon_bp_calc_ray_path +
// the atomic kernel, siddon_kernelsMLEM.cuh:307-365) to an accumulator whose z runs
// fastest, scaled for *top.  BANDS: nothing where the view is not of its band.  (The scale
// is worked out once a block, not once a ray: 64^3, 90 views, 3 us of 110.)
template <bool POW2, bool BANDS>
__device__ __forceinline__ void scatter_rays(float (*tile)[kRayRows + 1], const CompatGeom& G,
                                             const float* __restrict__ angles, const unsigned* __restrict__ loopN,
                                             unsigned view, VoxelStrides V, int u0, int v0,
                                             const float* __restrict__ img, const unsigned* __restrict__ maxabs,
                                             unsigned top, const BandRule& R, unsigned long long* acc)
{
    __shared__ double block_scale;
    const int t = threadIdx.y * kRayRows + threadIdx.x;
    {  // read eight columns (one 32-byte sector) at a time
        const int u = u0 + t % kRayCols, v = v0 + t / kRayCols;
        if (u < G.Nu && v < G.Nv) tile[t % kRayCols][t / kRayCols] = img[(size_t)u + (size_t)v * G.Nu];
    }
    if (t == 0) block_scale = (BANDS && !in_band(maxabs[view], top, R)) ? 0.0 : fix_scale(top, R.len_all, R.bits_all);
    __syncthreads();
    const int u = u0 + threadIdx.y, v = v0 + threadIdx.x;
    const double scale = block_scale;
    if (u >= G.Nu || v >= G.Nv || scale == 0.0) return;
    const float gi = tile[threadIdx.y][threadIdx.x];
    Ray r;
    setup(G, view_angle(angles, view), u, v, r);
    // scale is a power of two, so where FP32 holds it the product is exact there too
    // (or below the smallest normal, and rounds to 0 like the FP64 one)
    const float fscale = (float)scale;
    const bool single = scale >= 1e-30 && scale <= 1e30;
    walk<POW2>(G, r, loopN[view], V, [&](bool in, int id, float length) {
        const float c = __fmul_rn(length, gi);
        if (in && c != 0.0f) {
            const long long q = single ? __float2ll_rn(c * fscale) : __double2ll_rn((double)c * scale);
            if (q) atomicAdd(acc + id, (unsigned long long)q);
        }
    });
}

// Views view0 + blockIdx.y, view y reading img + y * img_stride, all scaled by
// maxabs[slot] (one view's bound, or the bound over all the views launched).  BANDS: the
// views of the band of maxabs[slot] only (maxabs[view] holding each view's own).
template <bool POW2, bool BANDS>
__global__ void __launch_bounds__(kRayRows * kRayCols, 4) bp_scatter_kernel(
    CompatGeom G, const float* __restrict__ angles, const unsigned* __restrict__ loopN, unsigned view0, VoxelStrides V,
    const float* __restrict__ img, size_t img_stride, const unsigned* __restrict__ maxabs, unsigned slot, BandRule R,
    unsigned long long* __restrict__ acc)
{
    __shared__ float tile[kRayCols][kRayRows + 1];
    const unsigned view = view0 + blockIdx.y;
    scatter_rays<POW2, BANDS>(tile, G, angles, loopN, view, V, blockIdx.x * kRayCols, blockIdx.z * kRayRows,
                              img + (size_t)blockIdx.y * img_stride, maxabs, maxabs[slot], R, acc);
}

// Fixed point -> float (one rounding), then out = v (overwrite) or
// out = out + v (siddon_add_bp into the running sum).  The accumulator's z runs fastest,
// the image's x: tile `xz` of 32 (x) x 32 (z) of one y, through shared memory.
// LOADS of a thread's four words in flight.
template <int LOADS>
__device__ __forceinline__ void finish_tile(float (*tile)[33], const unsigned long long* acc, int X, int Y, int Z, int xz,
                                            int y, double scale, float* out, bool accumulate)
{
    const double unscale = scale != 0.0 ? 1.0 / scale : 0.0;  // a power of two
    const int tx = (X + 31) / 32, x0 = xz % tx * 32, z0 = xz / tx * 32;
#pragma unroll 1
    for (int r = threadIdx.y; r < 32; r += 8 * LOADS) {
        unsigned long long q[LOADS];
#pragma unroll
        for (int k = 0; k < LOADS; ++k) {
            const int x = x0 + r + 8 * k, z = z0 + threadIdx.x;
            q[k] = (scale != 0.0 && x < X && z < Z) ? acc[((size_t)y * X + x) * Z + z] : 0ull;
        }
#pragma unroll
        for (int k = 0; k < LOADS; ++k) tile[r + 8 * k][threadIdx.x] = (float)((double)(long long)q[k] * unscale);
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += 8) {
        const int z = z0 + r, x = x0 + threadIdx.x;
        if (x < X && z < Z) {
            float* const o = out + ((size_t)z * Y + y) * X + x;
            *o = accumulate ? __fadd_rn(*o, tile[threadIdx.x][r]) : tile[threadIdx.x][r];
        }
    }
    __syncthreads();
}

__global__ void __launch_bounds__(256) bp_finish_kernel(const unsigned long long* __restrict__ acc, int X, int Y, int Z,
                                                        const unsigned* __restrict__ maxabs, unsigned view, float chord,
                                                        int count_bits, float* __restrict__ out, int accumulate)
{
    __shared__ float tile[32][33];
    const double scale = fix_scale(maxabs[view], chord, count_bits);
    for (int y = blockIdx.y; y < Y; y += gridDim.y)
        finish_tile<1>(tile, acc, X, Y, Z, (int)blockIdx.x, y, scale, out, accumulate != 0);
}

// The end of a back projection of several views: the first band's sums into out
// (overwritten, or added to), then, band by band from the brightest, the views that it left out, each
// band's sums added to out.  Sinograms whose views are of like magnitude have one band,
// and the kernel is then the finishing pass alone.  One cooperative launch, because only
// the device knows how many bands there are; every block works the bands out from the
// same maxima, so all of them take the same steps.
template <bool POW2>
__global__ void __launch_bounds__(kRayRows * kRayCols, 4) bp_bands_kernel(
    CompatGeom G, const float* __restrict__ angles, const unsigned* __restrict__ loopN, unsigned view0, unsigned views,
    VoxelStrides V, const float* __restrict__ img, const unsigned* __restrict__ maxabs, unsigned slot, BandRule R,
    unsigned long long* acc, float* out, int accumulate)
{
    __shared__ float tile[32][33];
    const int X = G.dims[0], Y = G.dims[1], Z = G.dims[2];
    const unsigned xz = (unsigned)((X + 31) / 32) * (unsigned)((Z + 31) / 32);
    const size_t nvox = (size_t)X * Y * Z, npix = (size_t)G.Nu * G.Nv, tiles = (size_t)xz * Y;
    const unsigned nu = (G.Nu + kRayCols - 1) / kRayCols, nv = (G.Nv + kRayRows - 1) / kRayRows;
    unsigned top = maxabs[slot];
    for (;; accumulate = 1) {
        const double scale = fix_scale(top, R.len_all, R.bits_all);
        for (size_t t = blockIdx.x; t < tiles; t += gridDim.x)
            finish_tile<4>(tile, acc, X, Y, Z, (int)(t % xz), (int)(t / xz), scale, out, accumulate != 0);
        top = next_band(maxabs + view0, views, top, R);
        if (top == 0u) return;
        cooperative_groups::this_grid().sync();  // the last band's sums are read
        for (size_t q = blockIdx.x * (size_t)256 + threadIdx.y * 32 + threadIdx.x; q < nvox; q += (size_t)gridDim.x * 256)
            acc[q] = 0ull;
        cooperative_groups::this_grid().sync();
        for (size_t b = blockIdx.x; b < (size_t)nu * nv * views; b += gridDim.x) {
            const unsigned n = (unsigned)(b / nu % views), view = view0 + n;
            if (!in_band(maxabs[view], top, R)) continue;
            scatter_rays<POW2, false>(reinterpret_cast<float (*)[kRayRows + 1]>(tile), G, angles, loopN, view, V,
                                      (int)(b % nu) * kRayCols, (int)(b / ((size_t)nu * views)) * kRayRows,
                                      img + (size_t)n * npix, maxabs, top, R, acc);
            __syncthreads();
        }
        cooperative_groups::this_grid().sync();
    }
}

// Clears the accumulator, n words of maxima and the word *top.
__global__ void __launch_bounds__(256) bp_clear_kernel(unsigned long long* __restrict__ acc, size_t nvox,
                                                       unsigned* maxabs, unsigned n, unsigned* top)
{
    const size_t t = blockIdx.x * (size_t)256 + threadIdx.x, stride = (size_t)gridDim.x * 256;
    for (size_t q = t; q < nvox; q += stride) acc[q] = 0ull;
    for (size_t q = t; q < n; q += stride) maxabs[q] = 0u;
    if (t == 0) *top = 0u;
}

// Each view's max |value| (float bits) into its cleared word, and into *top a bound on
// the finite views' (a view that is not finite may raise it; the bands after the first
// then take the views that this bound leaves out).
__global__ void __launch_bounds__(256) maxabs_views_kernel(const float* __restrict__ img, size_t npix,
                                                           unsigned* __restrict__ out, unsigned* __restrict__ top)
{
    const float* const a = img + (size_t)blockIdx.y * npix;
    unsigned m = 0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < npix; i += (size_t)gridDim.x * blockDim.x)
        m = max(m, __float_as_uint(fabsf(a[i])));
    m = __reduce_max_sync(0xffffffffu, m);
    __shared__ unsigned warps[8];
    if ((threadIdx.x & 31) == 0) warps[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x >= 32) return;
    m = __reduce_max_sync(0xffffffffu, warps[threadIdx.x & 7]);
    if (threadIdx.x != 0 || m == 0u) return;
    atomicMax(out + blockIdx.y, m);
    if (m < 0x7f800000u && m > *(volatile unsigned*)top) atomicMax(top, m);
}

// out = max over views of maxabs[0 .. n) (non-negative floats as unsigned bits)
__global__ void max_views_kernel(const unsigned* __restrict__ maxabs, unsigned n, unsigned* __restrict__ out)
{
    unsigned m = 0;
    for (unsigned i = threadIdx.x; i < n; i += blockDim.x) m = max(m, maxabs[i]);
    m = __reduce_max_sync(0xffffffffu, m);
    __shared__ unsigned w[32];
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned r = 0;
        for (unsigned k = 0; k < (blockDim.x + 31) / 32; ++k) r = max(r, w[k]);
        *out = r;
    }
}

}  // namespace compat

// ---- host side ---------------------------------------------------------------------

// Fewest views for which a forward projection makes the z-fastest copy of the volume:
// at 256^3 / 512^2 four views take 270 us without and 281 us with it, eight 458 and
// 436, sixteen 856 and 744 (64^3 and 128^3: within 3 us of each other from three on).
constexpr unsigned kZfastViews = 6;
constexpr int kZfastSlices = 32 * 65535;  // and most slices (launch_zfast's grid)

static dim3 ray_block() { return dim3(32, 4, 1); }
static dim3 ray_grid(const Plan& P, unsigned views)
{
    return dim3((P.cg.Nu + 31) / 32, (P.cg.Nv + 3) / 4, views);
}
static dim3 walk_block() { return dim3(compat::kRayRows, compat::kRayCols, 1); }
static dim3 walk_grid(const Plan& P, unsigned views)
{
    return dim3((P.cg.Nu + compat::kRayCols - 1) / compat::kRayCols, views,
                (P.cg.Nv + compat::kRayRows - 1) / compat::kRayRows);
}
static compat::VoxelStrides strides_x(const Plan& P) { return {1, P.cg.dims[0], P.cg.dims[0] * P.cg.dims[1]}; }
static compat::VoxelStrides strides_z(const Plan& P) { return {P.cg.dims[2], P.cg.dims[0] * P.cg.dims[2], 1}; }

// Voxel sizes that are powers of two: a division by one is an exact product.
static bool pow2_voxels(const Plan& P)
{
    for (float d : P.cg.Pd) {
        int e;
        if (std::frexp(d, &e) != 0.5f || e < -30 || e > 30) return false;
    }
    return true;
}

// Forward projections of plan views (or the scratch slot) from `first`.  From kZfastViews
// views on they read a copy of the volume whose z runs fastest, so that a warp's detector
// rows read neighbouring addresses; for fewer the copy costs more than it gives.  The copy
// goes to `scratch`, which belongs to the caller's own work, or without it to the plan's
// d_vol_z, which all calls on the plan share: an event orders those, so that calls on
// several streams stay independent.  A captured call, whose replays no event of the plan
// can order, reads the caller's volume instead.
template <int MODE>
static recon_status_t launch_compat_fp(Plan& P, unsigned first, unsigned count, const float* vol, const float* g,
                                       float* out, unsigned* maxabs, float* scratch, cudaStream_t s)
{
    if (count == 0) return RECON_OK;
    const bool wanted = count >= kZfastViews && P.cg.dims[2] <= kZfastSlices;
    float* copy = wanted ? scratch : nullptr;
    const bool shared = wanted && !scratch && P.d_vol_z;
    if (shared) {
        cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
        RB_CUDA(cudaStreamIsCapturing(s, &capturing));
        if (capturing == cudaStreamCaptureStatusNone) {
            copy = P.d_vol_z;
            RB_CUDA(cudaStreamWaitEvent(s, P.vol_z_free, 0));
        }
    }
    if (copy) RB_CHECK(launch_zfast(vol, copy, P.cg.dims[0], P.cg.dims[1], P.cg.dims[2], 0, s));
    auto kernel = pow2_voxels(P) ? compat::fp_kernel<MODE, true> : compat::fp_kernel<MODE, false>;
    note_kernel(RECON_PROJECTOR_FORWARD, "compat::fp_kernel");
    kernel<<<walk_grid(P, count), walk_block(), 0, s>>>(P.cg, P.d_angles, P.d_loopN, first,
                                                        copy ? strides_z(P) : strides_x(P), copy ? copy : vol, g, out,
                                                        maxabs);
    RB_CUDA(cudaGetLastError());
    if (copy && shared) RB_CUDA(cudaEventRecord(P.vol_z_free, s));
    return RECON_OK;
}

// The z-fastest copy's memory, for plans whose calls can use it; a plan that does not
// get it projects from the caller's volume.
recon_status_t compat_alloc_volume(Plan& P)
{
    if (P.nviews < kZfastViews || P.cg.dims[2] > kZfastSlices) return RECON_OK;
    if (P.alloc(&P.d_vol_z, P.nvox, "z-fastest volume") != RECON_OK) {
        P.d_vol_z = nullptr;
        return RECON_OK;
    }
    RB_CUDA(cudaEventCreateWithFlags(&P.vol_z_free, cudaEventDisableTiming));
    return RECON_OK;
}

static unsigned elem_blocks(size_t n) { return (unsigned)std::min<size_t>((n + 255) / 256, 148 * 16); }

// Back projections of `views` views from `first` into the cleared z-fastest accumulator,
// scaled by maxabs[slot] with the bounds of R for all of them; with bands, only the views
// of the first band.
static recon_status_t launch_scatter(Plan& P, unsigned first, unsigned views, const float* img, size_t img_stride,
                                     unsigned slot, const compat::BandRule& R, bool bands, cudaStream_t s)
{
    const bool pow2 = pow2_voxels(P);
    auto kernel = bands ? (pow2 ? compat::bp_scatter_kernel<true, true> : compat::bp_scatter_kernel<false, true>)
                        : (pow2 ? compat::bp_scatter_kernel<true, false> : compat::bp_scatter_kernel<false, false>);
    note_kernel(RECON_PROJECTOR_BACK, "compat::bp_scatter_kernel");
    kernel<<<walk_grid(P, views), walk_block(), 0, s>>>(P.cg, P.d_angles, P.d_loopN, first, strides_z(P), img, img_stride,
                                                        P.d_maxabs, slot, R, P.d_fix);
    RB_CUDA(cudaGetLastError());
    return RECON_OK;
}

// The accumulator, scaled by maxabs[slot], rounded once into out (overwritten, or added to).
static recon_status_t launch_finish(Plan& P, unsigned slot, float len, int bits, float* out, bool accumulate,
                                    cudaStream_t s)
{
    const int X = P.cg.dims[0], Y = P.cg.dims[1], Z = P.cg.dims[2];
    const dim3 grid((unsigned)((X + 31) / 32) * (unsigned)((Z + 31) / 32), std::min(Y, 65535));
    compat::bp_finish_kernel<<<grid, dim3(32, 8), 0, s>>>(P.d_fix, X, Y, Z, P.d_maxabs, slot, len, bits, out,
                                                          accumulate ? 1 : 0);
    RB_CUDA(cudaGetLastError());
    return RECON_OK;
}

// Upper bound of any source-to-pixel distance (every segment is part of one).
static float max_ray_length(const Plan& P)
{
    const recon_geometry_t& g = P.geom;
    double hu = 0.5 * g.det.NumAxPixels * (double)g.det.AxPixDimMm * std::fabs((double)g.cal.M) + std::fabs(g.cal.Dx);
    double hv = 0.5 * g.det.NumTAxPixels * (double)g.det.TAxPixDimMm * std::fabs((double)g.cal.M) + std::fabs(g.cal.Dz);
    double sc = std::fabs((double)g.cal.R) / std::max(1e-6, std::fabs((double)g.cal.Ry) - hu - hv);
    double R = std::fabs((double)g.cal.R) + std::fabs((double)g.cal.Rf);
    return (float)(2.0 * (R + sc * (hu + hv)) + 1.0);
}
static int count_bits(const Plan& P)
{
    int b = 0;
    while ((size_t(1) << b) < P.npix) ++b;
    return b + 1;
}

// Scale bounds for the sum over several views.  A segment
// lies on its ray between the volume's entry and exit, so it is no longer
// than the volume's diagonal.  A contribution to a voxel comes from a ray
// whose segment midpoint falls in it, i.e. a ray through the voxel's box (up
// to the index rounding): with an untilted detector those are the pixels in
// the box's shadow, at most W x H on the detector from the nearest depth the
// volume reaches, widened by three pixels each way, with at most four segments
// each.  A tilted detector falls back to one contribution per ray of the view.
static float volume_diagonal(const Plan& P)
{
    const recon_geometry_t& g = P.geom;
    const double x = g.vox.Xdim * (double)g.vox.XVoxSize, y = g.vox.Ydim * (double)g.vox.YVoxSize,
                 z = g.vox.Zdim * (double)g.vox.ZVoxSize;
    return (float)(std::sqrt(x * x + y * y + z * z) * 1.001 + 1e-3);
}

static int count_bits_all(const Plan& P, unsigned views)
{
    const recon_geometry_t& g = P.geom;
    double per_view = std::ldexp(1.0, count_bits(P));
    if (g.cal.xangle == 0.0f && g.cal.yangle == 0.0f && g.cal.zangle == 0.0f) {
        const double vx = std::fabs((double)g.vox.XVoxSize), vy = std::fabs((double)g.vox.YVoxSize),
                     vz = std::fabs((double)g.vox.ZVoxSize);
        const double rmax = 0.5 * std::hypot(g.vox.Xdim * vx, g.vox.Ydim * vy);
        const double dmin = std::fabs((double)g.cal.Rf) - rmax;
        const double pu = std::fabs((double)g.det.AxPixDimMm * g.cal.M), pv = std::fabs((double)g.det.TAxPixDimMm * g.cal.M);
        if (dmin > 0.0 && pu > 0.0 && pv > 0.0) {
            const double mag = std::max(std::fabs((double)g.cal.R), std::fabs((double)g.cal.Ry)) / dmin;
            const double diag = std::hypot(vx, vy), zmax = 0.5 * g.vox.Zdim * vz;
            const double W = diag * mag, H = (vz + diag * zmax / dmin) * mag;
            per_view = std::min(per_view, 4.0 * (std::ceil(W / pu) + 6.0) * (std::ceil(H / pv) + 6.0));
        }
    }
    const double total = per_view * std::max(1u, views);
    int b = 0;
    while (std::ldexp(1.0, b) < total) ++b;
    return b + 1;
}

__global__ void set_value_kernel(float* p, float v) { *p = v; }

static float* angles_dev(Plan& P) { return P.d_angles; }

recon_status_t build_compat_tables(Plan& P, cudaStream_t s)
{
    if (P.nviews == 0) return RECON_OK;
    RB_CUDA(cudaMemsetAsync(P.d_loopN, 0, (P.nviews + 1) * sizeof(unsigned), s));
    compat::loopn_kernel<<<ray_grid(P, P.nviews), ray_block(), 0, s>>>(P.cg, angles_dev(P), 0u, P.d_loopN);
    RB_CUDA(cudaGetLastError());
    return RECON_OK;
}

recon_status_t compat_view_loopN(Plan& P, float angle, unsigned slot, cudaStream_t s)
{
    float* ang = angles_dev(P);
    set_value_kernel<<<1, 1, 0, s>>>(ang + slot, angle);
    RB_CUDA(cudaMemsetAsync(P.d_loopN + slot, 0, sizeof(unsigned), s));
    compat::loopn_kernel<<<ray_grid(P, 1), ray_block(), 0, s>>>(P.cg, ang, slot, P.d_loopN);
    RB_CUDA(cudaGetLastError());
    return RECON_OK;
}

recon_status_t compat_fp(Plan& P, const float* vol, unsigned first, unsigned count, bool scratch_slot,
                         float angle_scratch, float* out, cudaStream_t s)
{
    if (scratch_slot) {
        RB_CHECK(compat_view_loopN(P, angle_scratch, P.nviews, s));
        first = P.nviews;
        count = 1;
    }
    return launch_compat_fp<0>(P, first, count, vol, nullptr, out, nullptr, nullptr, s);
}

// Back projection of one view, scaled by its own largest magnitude.
static recon_status_t compat_bp_into(Plan& P, const float* img, unsigned view, float* out, bool accumulate,
                                     cudaStream_t s)
{
    const compat::BandRule R{max_ray_length(P), max_ray_length(P), count_bits(P), count_bits(P)};
    compat::bp_clear_kernel<<<elem_blocks(P.nvox), 256, 0, s>>>(P.d_fix, P.nvox, P.d_maxabs + view, 1u,
                                                                  P.d_maxabs + view);
    RB_CUDA(cudaGetLastError());
    compat::maxabs_kernel<<<elem_blocks(P.npix), 256, 0, s>>>(img, P.npix, P.d_maxabs + view);
    RB_CUDA(cudaGetLastError());
    RB_CHECK(launch_scatter(P, view, 1, img, 0, view, R, false, s));
    return launch_finish(P, view, R.len, R.bits, out, accumulate, s);
}

recon_status_t compat_bp_view(Plan& P, const float* img, unsigned view, bool scratch_slot, float angle_scratch,
                              float* out, cudaStream_t s)
{
    if (scratch_slot) {
        RB_CHECK(compat_view_loopN(P, angle_scratch, P.nviews, s));
        view = P.nviews;
    }
    return compat_bp_into(P, img, view, out, false, s);
}

// Back projections of every plan view (view n's image at img + n * img_stride) summed in
// one 64-bit fixed-point accumulator, scaled by the bound over all of them
// (maxabs[nviews + 1], which the caller sets), and rounded to float once into out.  The
// reference adds each view's back projection into a float image
// (hf_siddon_recon.hpp:437-476); one rounding of the exact sum differs from that by float
// rounding only.
static recon_status_t compat_bp_all(Plan& P, const float* img, size_t img_stride, float* out, cudaStream_t s)
{
    const int bits = count_bits_all(P, P.nviews);
    const float len = volume_diagonal(P);
    RB_CUDA(cudaMemsetAsync(P.d_fix, 0, P.nvox * sizeof(unsigned long long), s));
    RB_CHECK(launch_scatter(P, 0u, P.nviews, img, img_stride, P.nviews + 1, compat::BandRule{len, len, bits, bits}, false, s));
    return launch_finish(P, P.nviews + 1, len, bits, out, false, s);
}

// Back projections of plan views first .. first + count - 1, at most as many as the bounds
// of R allow to share an accumulator, into out (overwritten, or added to).
static recon_status_t compat_bp_group(Plan& P, const float* sino, unsigned first, unsigned count,
                                      const compat::BandRule& rule, float* out, bool add, cudaStream_t s)
{
    unsigned* const maxima = P.d_maxabs + first;
    unsigned slot = P.nviews + 1;
    compat::bp_clear_kernel<<<elem_blocks(P.nvox), 256, 0, s>>>(P.d_fix, P.nvox, maxima, count,
                                                                  P.d_maxabs + slot);
    RB_CUDA(cudaGetLastError());
    const unsigned blocks = (unsigned)std::min<size_t>((P.npix + 1023) / 1024, 64);
    compat::maxabs_views_kernel<<<dim3(blocks, count), 256, 0, s>>>(sino, P.npix, maxima, P.d_maxabs + slot);
    RB_CUDA(cudaGetLastError());
    RB_CHECK(launch_scatter(P, first, count, sino, P.npix, slot, rule, true, s));
    compat::VoxelStrides V = strides_z(P);
    CompatGeom G = P.cg;
    compat::BandRule R = rule;
    const float* angles = P.d_angles;
    const unsigned *loopN = P.d_loopN, *maxabs = P.d_maxabs;
    unsigned long long* acc = P.d_fix;
    int accumulate = add ? 1 : 0;
    void* args[] = {&G, &angles, &loopN, &first, &count, &V, &sino, &maxabs, &slot, &R, &acc, &out, &accumulate};
    auto kernel = pow2_voxels(P) ? compat::bp_bands_kernel<true> : compat::bp_bands_kernel<false>;
    RB_CUDA(cudaLaunchCooperativeKernel((const void*)kernel, dim3(4 * P.sm_count), walk_block(), args, 0, s));
    return RECON_OK;
}

// Back projections of plan views first .. first + count - 1, summed.  Views share an
// accumulator, and are rounded to float together, where none of them loses a bit by it
// (bands, BandRule): 64^3, 90 views of like magnitude, 0.11 ms against 3.6 ms for a scatter
// and a finishing pass over the volume per view.  Views that are much dimmer than the
// brightest come in bands of their own; a view that holds a value that is not finite adds
// nothing, the others all they have.  Groups of views: as many as the bound for one view
// covers -- all of them with an untilted detector nearly always, 12 of 90 at 64^3 with a tilted
// one, for which there is no bound on the rays through a voxel but the detector's size.
recon_status_t compat_bp_views(Plan& P, const float* sino, unsigned first, unsigned count, float* out, cudaStream_t s)
{
    const compat::BandRule one{max_ray_length(P), volume_diagonal(P), count_bits(P), 0};
    // a magnitude's exponent under the one bound exceeds that under the other by at least this
    const int spare = (int)std::floor(std::log2((double)one.len / (double)one.len_all));
    unsigned group = count;
    while (group > 1 && count_bits_all(P, group) > one.bits + spare) group = (group + 1) / 2;
    for (unsigned n = 0; n < count; n += group) {
        const unsigned k = std::min(group, count - n);
        const float* const img = sino + (size_t)n * P.npix;
        if (k == 1) {
            RB_CHECK(compat_bp_into(P, img, first + n, out, n > 0, s));
            continue;
        }
        compat::BandRule R = one;
        R.bits_all = count_bits_all(P, k);
        RB_CHECK(compat_bp_group(P, img, first + n, k, R, out, n > 0, s));
    }
    return RECON_OK;
}

recon_status_t compat_sensitivity(Plan& P, float* sens, cudaStream_t s)
{
    if (P.nviews == 0) {
        RB_CUDA(cudaMemsetAsync(sens, 0, P.nvox * sizeof(float), s));
        return RECON_OK;
    }
    RB_CHECK(launch_fill(P.d_view_img, 1.0f, P.npix, s));
    set_value_kernel<<<1, 1, 0, s>>>(reinterpret_cast<float*>(P.d_maxabs + P.nviews + 1), 1.0f);
    RB_CUDA(cudaGetLastError());
    return compat_bp_all(P, P.d_view_img, 0, sens, s);
}

// m_mlem_single_iteration (hf_siddon_recon.hpp:437-476): FP and ratio of every
// view (the image is fixed within the iteration, so the views' order does not
// matter), the back projections of all ratios summed exactly, then
// f = f*Ht; f = divide1(f, sens).
recon_status_t compat_mlem_iteration(Plan& P, const float* g, float* f, cudaStream_t s)
{
    if (P.nviews == 0) return RECON_OK;
    RB_CUDA(cudaMemsetAsync(P.d_maxabs, 0, (P.nviews + 2) * sizeof(unsigned), s));
    float* ratio = static_cast<float*>(P.d_ratio);
    RB_CHECK(launch_compat_fp<1>(P, 0u, P.nviews, f, g, ratio, P.d_maxabs, P.d_ht, s));  // (Ht is written later)
    compat::max_views_kernel<<<1, 256, 0, s>>>(P.d_maxabs, P.nviews, P.d_maxabs + P.nviews + 1);
    RB_CUDA(cudaGetLastError());
    RB_CHECK(compat_bp_all(P, ratio, P.npix, P.d_ht, s));
    return launch_update(f, P.d_ht, P.d_sens, P.nvox, true, s);
}

// divide1(g, FP(f)) for every view, into a full ratio sinogram (input of the
// voxel-driven back projector).
recon_status_t compat_fp_ratio_all(Plan& P, const float* vol, const float* g, float* ratio, cudaStream_t s)
{
    RB_CUDA(cudaMemsetAsync(P.d_maxabs, 0, (P.nviews + 1) * sizeof(unsigned), s));
    return launch_compat_fp<1>(P, 0u, P.nviews, vol, g, ratio, P.d_maxabs, P.d_ht, s);  // (no other use of Ht here)
}

// ---- parity entry points --------------------------------------------------------------

recon_status_t compat_setup_dump(Plan& P, float angle, float* h[10], unsigned* loopN)
{
    cudaStream_t s = 0;
    const size_t n = P.npix;
    float *amin, *amax, *d12, *ai, *af, *da, *p1, *p2;
    unsigned *mask, *dindex;
    size_t bytes = n * (3 * 4 + 4 + 4 + 5 * 12) + 16;
    char* base = nullptr;
    RB_CUDA(cudaMalloc(&base, bytes));
    char* q = base;
    auto take = [&](size_t b) { char* r = q; q += b; return r; };
    amin = (float*)take(n * 4); amax = (float*)take(n * 4); d12 = (float*)take(n * 4);
    mask = (unsigned*)take(n * 4); ai = (float*)take(n * 12); af = (float*)take(n * 12);
    da = (float*)take(n * 12); p1 = (float*)take(n * 12); p2 = (float*)take(n * 12);
    dindex = (unsigned*)take(n * 4);
    compat::setup_dump_kernel<<<ray_grid(P, 1), ray_block(), 0, s>>>(P.cg, angle, amin, amax, d12, mask, ai, af, da,
                                                                      p1, p2, dindex);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(cudaStreamLegacy);
    void* dev[10] = {amin, amax, d12, mask, ai, af, da, p1, p2, dindex};
    size_t sz[10] = {n * 4, n * 4, n * 4, n * 4, n * 12, n * 12, n * 12, n * 12, n * 12, n * 4};
    for (int k = 0; k < 10 && e == cudaSuccess; ++k) e = cudaMemcpy(h[k], dev[k], sz[k], cudaMemcpyDeviceToHost);
    cudaFree(base);
    if (e != cudaSuccess) return cuda_fail(e, "compat setup dump");
    unsigned mx = 0;
    const unsigned* di = reinterpret_cast<const unsigned*>(h[9]);
    for (size_t i = 0; i < n; ++i) mx = std::max(mx, di[i]);
    *loopN = mx;
    return RECON_OK;
}

recon_status_t compat_trace(Plan& P, float angle, int nrays, const int* rays, int cap, int* idx, float* len,
                            unsigned* loopN_out)
{
    RB_CHECK(compat_view_loopN(P, angle, P.nviews, 0));
    unsigned loopN = 0;
    RB_CUDA(cudaMemcpy(&loopN, P.d_loopN + P.nviews, sizeof(unsigned), cudaMemcpyDeviceToHost));
    int *d_rays = nullptr, *d_idx = nullptr;
    float* d_len = nullptr;
    cudaError_t e = cudaMalloc(&d_rays, sizeof(int) * std::max(1, nrays));
    if (e == cudaSuccess) e = cudaMalloc(&d_idx, sizeof(int) * (size_t)std::max(1, nrays) * cap);
    if (e == cudaSuccess) e = cudaMalloc(&d_len, sizeof(float) * (size_t)std::max(1, nrays) * cap);
    if (e == cudaSuccess) e = cudaMemcpy(d_rays, rays, sizeof(int) * nrays, cudaMemcpyHostToDevice);
    if (e == cudaSuccess && nrays > 0) {
        compat::trace_kernel<<<(nrays + 127) / 128, 128>>>(P.cg, angle, loopN, nrays, d_rays, cap, d_idx, d_len);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaStreamSynchronize(cudaStreamLegacy);
        if (e == cudaSuccess) e = cudaMemcpy(idx, d_idx, sizeof(int) * (size_t)nrays * cap, cudaMemcpyDeviceToHost);
        if (e == cudaSuccess) e = cudaMemcpy(len, d_len, sizeof(float) * (size_t)nrays * cap, cudaMemcpyDeviceToHost);
    }
    cudaFree(d_rays);
    cudaFree(d_idx);
    cudaFree(d_len);
    if (e != cudaSuccess) return cuda_fail(e, "compat trace");
    *loopN_out = loopN;
    return RECON_OK;
}

}  // namespace rb
