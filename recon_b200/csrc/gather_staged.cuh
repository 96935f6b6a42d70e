// gather_staged.cuh -- what the staged gather (gather_staged.cu) and the few-view one
// (gather_few.cu) share, and the staged one's tile of voxel columns, its loads by TMA and
// their barriers, and the detector columns and rows it needs.
#pragma once

#include "gather_device.cuh"

#include <cudaTypedefs.h>

namespace rb {
namespace exact {

// A CTA owns a tile of TX x TY voxel columns, one warp each, and one more warp loads.
constexpr int kStagedTX = 4, kStagedTY = 4;
constexpr int kStagedWarps = kStagedTX * kStagedTY;
constexpr int kStagedThreads = (kStagedWarps + 1) * 32;

// What a stage holds and how columns meet the detector, from the host (staged_shape).
struct StagedShape {
    int rows;     // staged row pairs per detector column (multiple of 4): the box's width
    int cols;     // staged detector columns per view: the box's height
    int wide;     // most detector columns one voxel column meets in a view: 1, 2, 4 or 8
};

// One detector column of one view as a voxel column sees it: the piece [A, B] of
// its rays, row coefficients ca = ez / (A + Rf), cb = ez / (B + Rf), their steps
// per slot (32 voxels) pa, pb, and the detector column u; one = no voxel of the
// column has a second candidate row there.
struct StagedItem {
    float A, B, pa, pb, ca, cb;
    int u, one;
};

// ---- bulk copies and their barriers --------------------------------------------------------

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned bar)
{
    asm volatile("{\n\t.reg .b64 t;\n\tmbarrier.arrive.shared::cta.b64 t, [%0];\n\t}" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned bar, unsigned bytes)
{
    asm volatile("{\n\t.reg .b64 t;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 t, [%0], %1;\n\t}" ::"r"(bar),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try(unsigned bar, unsigned parity)
{
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity), "r"(1000000u)  // the warp may sleep up to 1 ms (ns) in one try
        : "memory");
    return done != 0u;
}
// Waits until the barrier's phase of this parity is complete; gives up after `limit` clocks
// (false), by default about two seconds, which no run that works comes near.
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity, long long limit = 4000000000ll)
{
    if (mbar_try(bar, parity)) return true;
    const long long t0 = clock64();
    while (!mbar_try(bar, parity))
        if (clock64() - t0 > limit) return false;
    return true;
}
// A wait was given up: the plan's word in host memory says so to its next call.
__device__ __forceinline__ void report_give_up(unsigned* word)
{
    *(volatile unsigned*)word = 1u;
    __threadfence_system();
}
// The box at entry x (a multiple of four) of table row y into dst (128-byte aligned).
__device__ __forceinline__ void tile_load(unsigned dst, const CUtensorMap* map, int x, int y, unsigned bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            dst),
        "l"(map), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

// a += L * x in both halves: one packed instruction, each half rounded as fmaf.
__device__ __forceinline__ void fma_pair(float2& a, float L, float2 x)
{
    unsigned long long acc = *reinterpret_cast<unsigned long long*>(&a);
    const unsigned long long v = *reinterpret_cast<const unsigned long long*>(&x);
    asm("{\n\t.reg .b64 l;\n\tmov.b64 l, {%1, %1};\n\tfma.rn.f32x2 %0, l, %2, %0;\n\t}" : "+l"(acc) : "f"(L), "l"(v));
    a = *reinterpret_cast<float2*>(&acc);
}

// Reads of shared memory at 32-bit addresses: a pair as stored (widen_lo / widen_hi
// give its values), a row's z planes.
__device__ __forceinline__ float2 lds_pair(unsigned a, float)
{
    float2 p;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(p.x), "=f"(p.y) : "r"(a));
    return p;
}
__device__ __forceinline__ unsigned lds_pair(unsigned a, __nv_bfloat16)
{
    unsigned p;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(p) : "r"(a));
    return p;
}
__device__ __forceinline__ float4 lds_planes(unsigned a)
{
    float4 p;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(p.x), "=f"(p.y), "=f"(p.z), "=f"(p.w) : "r"(a));
    return p;
}

// The rows that heights [zb, zt] are seen at from depths [dmin, dmax], widened by one row on
// either side.
__device__ __forceinline__ void staged_rows(const GatherConst& C, float zb, float zt, float dmin, float dmax,
                                            float& lo, float& hi)
{
    const float b0 = zb / dmin * C.ez, b1 = zb / dmax * C.ez, t0 = zt / dmin * C.ez, t1 = zt / dmax * C.ez;
    lo = fminf(b0, b1) + C.oz - 1.0f;
    hi = fmaxf(t0, t1) + C.oz + 1.0f;
}

// The first detector column that the rectangle [Xa, Xb] x [Ya, Yb] shadows at a view;
// the columns that staged_item gives a voxel column inside it start there or later.
__device__ __forceinline__ int staged_first_column(const ExactGeom& G, const GatherConst& C, const float2 CS, float Xa,
                                                   float Xb, float Ya, float Yb)
{
    float umin = 3.0e38f;
#pragma unroll
    for (int c4 = 0; c4 < 4; ++c4) {
        const float X = (c4 & 1) ? Xb : Xa, Y = (c4 & 2) ? Yb : Ya;
        const float a = X * CS.x - Y * CS.y, b = X * CS.y + Y * CS.x;
        umin = fminf(umin, __fdividef(a, b + G.Rf) * C.eu + C.ou);
    }
    return min(max(0, __float2int_ru(umin - 0.02f)), G.Nu - 1);
}

// Voxel column (i, j)'s item for detector column number sl of its range at a view;
// valid when it returns true.
__device__ __forceinline__ bool staged_item(const ExactGeom& G, const GatherConst& C, const float4* __restrict__ txy,
                                            const int2* __restrict__ kxy, const float2 CS, unsigned view, int sl, int i,
                                            int j, float Xa, float Xb, float Ya, float Yb, float margin, float dz32,
                                            StagedItem& it)
{
    float umin = 3.0e38f, umax = -3.0e38f;
#pragma unroll
    for (int c4 = 0; c4 < 4; ++c4) {
        const float X = (c4 & 1) ? Xb : Xa, Y = (c4 & 2) ? Yb : Ya;
        const float a = X * CS.x - Y * CS.y, b = X * CS.y + Y * CS.x;
        const float uf = __fdividef(a, b + G.Rf) * C.eu + C.ou;
        umin = fminf(umin, uf);
        umax = fmaxf(umax, uf);
    }
    const int u_lo = min(max(0, __float2int_ru(umin - 0.01f)), G.Nu);
    const int u_hi = min(G.Nu - 1, __float2int_rd(umax + 0.01f));
    it.u = u_lo + sl;
    if (it.u > u_hi) return false;
    const float4 T = __ldg(txy + (size_t)view * G.Nu + it.u);
    const int2 K = __ldg(kxy + (size_t)view * G.Nu + it.u);
    const float xa = plane_t(i, T.x, T.y, K.x), xb = plane_t(i + 1, T.x, T.y, K.x);
    const float ya = plane_t(j, T.z, T.w, K.y), yb = plane_t(j + 1, T.z, T.w, K.y);
    it.A = fmaxf(fminf(xa, xb), fminf(ya, yb));
    it.B = fminf(fmaxf(xa, xb), fmaxf(ya, yb));
    if (!(it.A < it.B)) return false;
    it.ca = __fdividef(C.ez, it.A + G.Rf);
    it.cb = __fdividef(C.ez, it.B + G.Rf);
    it.pa = dz32 * it.ca;
    it.pb = dz32 * it.cb;
    // a voxel's candidate interval has a length convex in its height, largest at
    // the column's bottom or top voxel
    const float zb = G.P0[2], zt = G.P0[2] + (float)G.Z * G.vox[2];
    const float len_b = fmaxf((zb + G.vox[2]) * it.ca, (zb + G.vox[2]) * it.cb) - fminf(zb * it.ca, zb * it.cb);
    const float len_t = fmaxf(zt * it.ca, zt * it.cb) - fminf((zt - G.vox[2]) * it.ca, (zt - G.vox[2]) * it.cb);
    it.one = (fmaxf(len_b, len_t) + margin < 0.99f) ? 1 : 0;
    return true;
}

}  // namespace exact

// Dynamic shared memory that a staged gather may use: a block's, less the items, the
// barriers and the base's alignment.
constexpr size_t kStagedSmem = 227 * 1024 - sizeof(exact::StagedItem) * 32 * exact::kStagedWarps - 1536;

int staged_wide(const Plan& P);
bool several_candidate_rows(const Plan& P);

}  // namespace rb
