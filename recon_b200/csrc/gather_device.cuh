// gather_device.cuh -- device functions shared by the gather back projectors
// (exact.cu, gather_staged.cu): a voxel column's rays seen from one view.
#pragma once

#include "exact_device.cuh"

namespace rb {
namespace exact {

struct GatherConst {
    float eu, ou;  // detector column of a point (a, b) of the view frame: a / (b + Rf) * eu + ou
    float ez, oz;  // detector row of height z at depth d (t = d - Rf):      z / d * ez + oz
    int vec4;      // X % 4 == 0 and the volume, sensitivity 16-byte aligned: float4 epilogue
};

// MLEM update of one voxel, as update_kernel computes it
__device__ __forceinline__ float gather_update(float f, float ht, float sens)
{
    return (sens != 0.0f) ? __fdiv_rn(__fmul_rn(f, ht), sens) : 0.0f;
}

// A warp's column seen from one view: detector columns u_lo..u_hi and, for the
// first two (sl = 0, 1), the column's piece [A, B] of their rays, the row
// coefficients ca = ez / (A + Rf), cb = ez / (B + Rf) and the per-slot steps
// pa = 32 vz ca, pb = 32 vz cb of the row bounds.  flags: bit sl = the rays of
// u_lo + sl cross the column (A < B); bit 2 + sl = no voxel of the column has
// a second candidate row there; bit 4 + sl = the piece lies behind the source
// (every row is a candidate).
struct GatherView {
    float4 ab[2];  // {A, B, pa, pb}
    float2 c[2];   // {ca, cb}
    int u_lo, u_hi;
    unsigned flags;
    unsigned view;  // the view's index (fills the struct's 16-byte alignment)
};

// Column (i, j) of the volume, [Xa, Xb] x [Ya, Yb], seen from one view (see
// GatherView); margin = the candidate rows' total widening (0.004 row).
__device__ __forceinline__ GatherView gather_view(const ExactGeom& G, const GatherConst& C,
                                                  const float4* __restrict__ txy, const int2* __restrict__ kxy,
                                                  const float2* __restrict__ cs, unsigned view, int i, int j, float Xa,
                                                  float Xb, float Ya, float Yb, float margin, float dz32)
{
    const float2 CS = __ldg(cs + view);
    float umin = 3.0e38f, umax = -3.0e38f;
    bool behind = false;
#pragma unroll
    for (int c4 = 0; c4 < 4; ++c4) {
        const float X = (c4 & 1) ? Xb : Xa, Y = (c4 & 2) ? Yb : Ya;
        const float a = X * CS.x - Y * CS.y, b = X * CS.y + Y * CS.x;
        const float d = b + G.Rf;
        behind |= !(d > 1e-3f * G.Rf);
        const float uf = a / d * C.eu + C.ou;
        umin = fminf(umin, uf);
        umax = fmaxf(umax, uf);
    }
    GatherView V;
    V.flags = 0u;
    V.view = view;
    if (behind) {  // not for a volume in front of the source; stays exact anyway
        V.u_lo = 0;
        V.u_hi = G.Nu - 1;
    } else {
        V.u_lo = min(max(0, __float2int_ru(umin - 0.01f)), G.Nu);
        V.u_hi = min(G.Nu - 1, __float2int_rd(umax + 0.01f));
    }
#pragma unroll
    for (int sl = 0; sl < 2; ++sl) {
        const int u = min(V.u_lo + sl, G.Nu - 1);
        const float4 T = __ldg(txy + (size_t)view * G.Nu + u);
        const int2 K = __ldg(kxy + (size_t)view * G.Nu + u);
        const float xa = plane_t(i, T.x, T.y, K.x), xb = plane_t(i + 1, T.x, T.y, K.x);
        const float ya = plane_t(j, T.z, T.w, K.y), yb = plane_t(j + 1, T.z, T.w, K.y);
        const float A = fmaxf(fminf(xa, xb), fminf(ya, yb));
        const float B = fminf(fmaxf(xa, xb), fmaxf(ya, yb));
        const float ca = C.ez / (A + G.Rf), cb = C.ez / (B + G.Rf);
        V.ab[sl] = make_float4(A, B, dz32 * ca, dz32 * cb);
        V.c[sl] = make_float2(ca, cb);
        if (A < B) V.flags |= 1u << sl;
        // a voxel's candidate interval [f0, f1] (row units) has a length
        // convex in its height, largest at the column's bottom or top voxel
        const float zb = G.P0[2], zt = G.P0[2] + (float)G.Z * G.vox[2];
        const float len_b = fmaxf((zb + G.vox[2]) * ca, (zb + G.vox[2]) * cb) - fminf(zb * ca, zb * cb);
        const float len_t = fmaxf(zt * ca, zt * cb) - fminf((zt - G.vox[2]) * ca, (zt - G.vox[2]) * cb);
        if (fmaxf(len_b, len_t) + margin < 0.99f) V.flags |= 1u << (2 + sl);
        if (!(A + G.Rf > 1e-3f * G.Rf)) V.flags |= 1u << (4 + sl);
    }
    return V;
}

}  // namespace exact

exact::GatherConst gather_const(const Plan& P, const float* vol, const float* sens);
// gather_staged.cu
template <int EPI, class ST>
recon_status_t staged_quarter_gather(Plan& P, const ST* vals, size_t view_stride, float* vol, const float* sens,
                                     cudaStream_t s, unsigned long long* npairs, bool set, unsigned m0, unsigned mc,
                                     bool* served);
// gather_few.cu
recon_status_t few_views_gather(Plan& P, const float* vals, size_t view_stride, unsigned first, unsigned count, float* vol,
                                cudaStream_t s, bool* served);

}  // namespace rb
