// gather_few.cu -- the mirror-paired gather back projector for a few views.
//
// The gathers that give a warp one voxel column set its views up one per lane; with one
// view a warp sets up one, and its chain of dependent loads (view, table, value, image) is
// all it does.  Here a warp owns eight columns along x: its lanes set them up (four sets of
// a view and a detector column at a time), the warp then gathers column after column, and
// the eight are staged so that the image is written in whole sectors.  Lengths and values
// are bp_gather_pairs_kernel's, and so is the order where a voxel has one candidate row per
// detector column and view; that kernel sums further candidates apart, this one in place.
//
// Bound by the latency of a warp's columns, one after the other (a load from L2 each).
// 256^3 / 512^2, one view: see few_views_suit for both sides.
#include "gather_staged.cuh"

#include <algorithm>
#include <type_traits>

namespace rb {
namespace exact {

constexpr int kFewWarps = 4;  // rows (y) of eight columns per CTA
constexpr int kFewStage = 8;  // columns of a warp

// Views view0 .. view0 + nview - 1, vals in mirrored row pairs (view_stride elements per
// view), vol overwritten.  wide: most detector columns that a voxel column meets in a view.
// Dynamic shared memory: the lower rows' z planes, then per warp its items
// [view][wide][column] and their masks.
template <int PS>
__global__ void __launch_bounds__(kFewWarps * 32, 4) bp_gather_few_kernel(
    ExactGeom G, GatherConst C, int wide, const float4* __restrict__ txy, const int2* __restrict__ kxy,
    const float2* __restrict__ cs, const ZParam* __restrict__ zp, unsigned view0, int nview,
    const float* __restrict__ vals, size_t view_stride, float* __restrict__ vol)
{
    extern __shared__ float4 szq[];
    constexpr int NE = 2 * PS * 32, NP = NE + 4;  // a staged column, padded against bank conflicts
    __shared__ float stage[kFewWarps][kFewStage][NP];
    const int Nh = G.Nv / 2, Zh = G.Z / 2;
    const int sets = nview * wide;
    StagedItem* const items0 = reinterpret_cast<StagedItem*>(szq + Nh + 1);
    unsigned* const masks0 = reinterpret_cast<unsigned*>(items0 + (size_t)kFewWarps * sets * kFewStage);
    const int nmask = (sets + 3) / 4;  // one word per four sets, eight bits each
    for (int q = threadIdx.x; q <= Nh; q += blockDim.x) {
        const ZParam z = zp[q];
        const float kc = (float)z.kc;
        szq[q] = (z.S > 0.0f) ? make_float4(z.S, z.O, kc, kc - 1.0f) : make_float4(z.S, z.O, kc - 1.0f, kc);
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i0 = blockIdx.x * kFewStage, i = i0 + lane % kFewStage, j = blockIdx.y * kFewWarps + warp;
    StagedItem* const items = items0 + (size_t)warp * sets * kFewStage;
    unsigned* const masks = masks0 + warp * nmask;
    const float oz_lo = C.oz - 0.002f, oz_hi = C.oz + 0.002f;  // margins as in bp_gather_kernel
    const float dz32 = 32.0f * G.vox[2];
    if (j < G.Y) {
        const float Xa = G.P0[0] + i * G.vox[0], Xb = Xa + G.vox[0];
        const float Ya = G.P0[1] + j * G.vox[1], Yb = Ya + G.vox[1];
        for (int t = 0; t < nmask; ++t) {
            const int set = 4 * t + lane / kFewStage;
            bool valid = false;
            if (set < sets && i < G.X) {
                const unsigned m = view0 + set / wide;
                StagedItem it;
                valid = staged_item(G, C, txy, kxy, __ldg(cs + m), m, set % wide, i, j, Xa, Xb, Ya, Yb, oz_hi - oz_lo, dz32,
                                    it);
                if (valid) items[set * kFewStage + lane % kFewStage] = it;
            }
            const unsigned bits = __ballot_sync(0xffffffffu, valid);
            if (lane == 0) masks[t] = bits;
        }
    }
    __syncthreads();
    if (j >= G.Y) return;  // whole warps; no barrier follows
    const int Np = pair_entries(G.Nv);
    const size_t plane = (size_t)G.X * G.Y;
    for (int k0 = 0; k0 < Zh; k0 += 32 * PS) {
        const float fk0 = (float)(k0 + lane);
        const float zl0 = fmaf(fk0, G.vox[2], G.P0[2]), zh0 = zl0 + G.vox[2];
        for (int c = 0; c < kFewStage; ++c) {
            float2 acc[PS];
#pragma unroll
            for (int s = 0; s < PS; ++s) acc[s] = make_float2(0.0f, 0.0f);
            for (int w = 0; w < sets; ++w) {
                if (!((masks[w >> 2] >> ((w & 3) * kFewStage + c)) & 1u)) continue;  // (the same for the warp)
                const StagedItem I = items[w * kFewStage + c];
                const float* const col =
                    vals + (size_t)(wide == 1 ? w : w / wide) * view_stride + (size_t)I.u * Np * 2;
                auto length = [&](int s, int v) {
                    const float4 zr = szq[v];
                    const float t = fk0 + (float)(32 * s);
                    const float lo = fmaf(t - zr.z, zr.x, zr.y), hi = fmaf(t - zr.w, zr.x, zr.y);
                    return fminf(I.B, hi) - fmaxf(I.A, lo);
                };
                const float P0a = fmaf(zl0, I.ca, oz_lo);
                int a[PS];
                float2 x[PS];
#pragma unroll
                for (int s = 0; s < PS; ++s) {
                    a[s] = (int)min(__float2uint_ru(fmaf((float)s, I.pa, P0a)), (unsigned)Nh);
                    x[s] = __ldg(reinterpret_cast<const float2*>(col + 2 * a[s]));
                }
#pragma unroll
                for (int s = 0; s < PS; ++s) {
                    const float L = length(s, a[s]);
                    if (L > 0.0f) {
                        acc[s].x = fmaf(L, x[s].x, acc[s].x);
                        acc[s].y = fmaf(L, x[s].y, acc[s].y);
                    }
                }
                if (I.one) continue;
                // further candidate rows, over the bounds of both piece ends
                const float P0b = fmaf(zl0, I.cb, oz_lo), P1a = fmaf(zh0, I.ca, oz_hi), P1b = fmaf(zh0, I.cb, oz_hi);
#pragma unroll
                for (int s = 0; s < PS; ++s) {
                    const float f0 = fminf(fmaf((float)s, I.pa, P0a), fmaf((float)s, I.pb, P0b));
                    const float f1 = fmaxf(fmaf((float)s, I.pa, P1a), fmaf((float)s, I.pb, P1b));
                    const int b = min(Nh, __float2int_rd(f1));
                    for (int v = max(0, __float2int_ru(f0)); v <= b; ++v) {
                        if (v == a[s]) continue;
                        const float L = length(s, v);
                        if (!(L > 0.0f)) continue;
                        const float2 y = __ldg(reinterpret_cast<const float2*>(col + 2 * v));
                        acc[s].x = fmaf(L, y.x, acc[s].x);
                        acc[s].y = fmaf(L, y.y, acc[s].y);
                    }
                }
            }
            float* const o = stage[warp][c];
#pragma unroll
            for (int s = 0; s < PS; ++s) {
                o[s * 32 + lane] = acc[s].x;
                o[(PS + s) * 32 + lane] = acc[s].y;
            }
        }
        __syncwarp();
        // eight columns of one slice (a sector) per eight lanes
        const int x = lane % kFewStage;
        for (int e = lane / kFewStage; e < NE; e += 32 / kFewStage) {
            const int k = k0 + e % (32 * PS);
            if (k >= Zh || i0 + x >= G.X) continue;
            const int z = e < 32 * PS ? k : G.Z - 1 - k;
            vol[(size_t)z * plane + (size_t)j * G.X + (size_t)(i0 + x)] = stage[warp][x][e];
        }
        __syncwarp();
    }
}

}  // namespace exact

// ---- host side -----------------------------------------------------------------------------

constexpr size_t kFewSmem = 64 * 1024;  // dynamic shared memory of the few-view kernel, at most

static size_t few_smem(const Plan& P, unsigned count, int wide)
{
    const size_t sets = (size_t)count * wide;
    return (size_t)(P.eg.Nv / 2 + 1) * sizeof(float4) +
           exact::kFewWarps * (sets * exact::kFewStage * sizeof(exact::StagedItem) + (sets + 3) / 4 * sizeof(unsigned));
}

// The few-view kernel's side of the line against bp_gather_pairs_kernel: enough columns
// (x, y) to share its warps' latency.  us with and without it, layout included; rows a voxel
// apart (AUTO's gather): 80^3 one view 15 and 14, 96^3 one 15 and 17, two 17 and 17, 96 x 96
// x 300 22 and 26, 27 and 29, 48 x 48 x 300 21 and 14, 25 and 15; 128^3 one to four 15 19 23 28
// and 23 25 27 30; 256^3 47 58 73 98 and 82 95 107 119.  Closer rows, of which voxels have
// several: 96^3 one 19 and 20, 96 x 96 x 160 23 and 21, 112^3 21 and 23, 112 x 112 x 300 38 and 39; two views
// 128^3 29 and 33, 160^3 62 and 56 (800 CTAs, a round and a third), 200^3 80 and 88, 256^3 130
// and 146; three 128^3 43 and 39, 256^3 194 and 183 (but 200 x 200 x 64 49 and 64, four 62 and
// 74: up to 64 slices the same line as for rows a voxel apart).
static int few_views_suit(const Plan& P, unsigned count)
{
    const ExactGeom& E = P.eg;
    const size_t columns = (size_t)E.X * E.Y;
    if (!P.col_pairs || count == 0 || count > 4) return 0;
    if (E.Z > 64 && several_candidate_rows(P)) {
        const int ctas = ((E.X + exact::kFewStage - 1) / exact::kFewStage) * ((E.Y + exact::kFewWarps - 1) / exact::kFewWarps);
        if (count > 2 || columns < (E.Z <= 128 ? 9216u : 12544u)) return 0;
        if (count == 2 && (columns < 16384 || (ctas > 4 * P.sm_count && ctas < 8 * P.sm_count))) return 0;
    } else if (columns < (count <= 2 ? 9216u : 16384u)) {
        return 0;
    }
    const int wide = staged_wide(P);
    return wide > 0 && wide <= 4 && few_smem(P, count, wide) <= kFewSmem ? wide : 0;
}

// Back projection of table slots first .. first + count - 1 from mirrored row pairs;
// *served = false (and nothing launched) where the gathers of exact.cu are to.
recon_status_t few_views_gather(Plan& P, const float* vals, size_t view_stride, unsigned first, unsigned count, float* vol,
                                cudaStream_t s, bool* served)
{
    const int wide = few_views_suit(P, count);
    *served = wide > 0;
    if (!*served) return RECON_OK;
    const ExactGeom& E = P.eg;
    const size_t smem = few_smem(P, count, wide);
    const dim3 grid((E.X + exact::kFewStage - 1) / exact::kFewStage, (E.Y + exact::kFewWarps - 1) / exact::kFewWarps);
    auto run = [&](auto ps) -> recon_status_t {
        auto kernel = exact::bp_gather_few_kernel<decltype(ps)::value>;
        RB_CHECK(allow_dynamic_smem(kernel, kFewSmem));
        note_kernel(RECON_PROJECTOR_BACK, "bp_gather_few_kernel");
        kernel<<<grid, exact::kFewWarps * 32, smem, s>>>(E, gather_const(P, vol, nullptr), wide, P.d_txy, P.d_kxy, P.d_cs,
                                                         P.d_zp, first, (int)count, vals, view_stride, vol);
        RB_CUDA(cudaGetLastError());
        return RECON_OK;
    };
    const int half = E.Z / 2;
    if (half <= 32) return run(std::integral_constant<int, 1>{});
    if (half <= 64) return run(std::integral_constant<int, 2>{});
    return run(std::integral_constant<int, 4>{});
}

}  // namespace rb
