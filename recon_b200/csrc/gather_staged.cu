// gather_staged.cu -- the EXACT gather back projector with its values staged in
// shared memory by TMA.
//
// The gathers of exact.cu read each candidate row's value from L2 where they use
// it, and a warp that owns a voxel column in registers leaves few warps to cover
// that latency.  Here a CTA owns a tile of columns (one warp each) and one more
// warp streams in what the tile reads: for every view the few detector columns
// that the tile's shadow covers, cropped to the rows that its slices can meet
// (one TMA box per view, completion on an mbarrier).  The column warps then find
// every value in shared memory at 32-bit addresses.
//
// Measured (256^3, 360 views, 512^2; one B200): 1.56 ms against
// bp_gather_quarter_kernel's 2.41 ms; 512^3, 720 views, 1024 x 768, BF16 ratio:
// 22.8 against 40.2 ms.  Bound by shared-memory reads (77 % of the wavefront peak:
// 0.34e9 wavefronts, 68 for 1024 products) with 0.94e9 warp instructions (1.56e9).
// What brought it there: loading the columns one by one with untiled bulk copies 3.46 ms
// (28 copies a view, the loading warp the limit), TMA boxes 2.10, two or four views to a
// stage instead of one 1.75, packed multiply-adds without a predicate 1.56.  Reading the
// zero entry of a region in place of the predicate cost bank conflicts (2.05).
#include "gather_staged.cuh"

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace rb {
namespace exact {

// ---- the quarter-turn gather ----------------------------------------------------------------

// bp_gather_quarter_kernel's sums (see there: one warp per base column of the
// quadrant x, y < X/2, every length found at view m serving the voxel pair in the
// four columns of its orbit at views m + rQ), in the same order, so the same bits.
// A CTA owns TX x TY base columns (kWarps warps) and a loading warp; a stage holds
// the four views' values of one base view, [r][detector column][row pair].
constexpr int kStageBytes = 98304;  // a stage: two or four base views of four regions of 12 or 6 KiB
constexpr unsigned kStages = 2;     // what a block's shared memory holds

template <int EPI, class ST, int PS, int RB, bool SET>
__global__ void __launch_bounds__(kStagedThreads, 1) bp_staged_quarter_kernel(
    ExactGeom G, GatherConst C, StagedShape S, const float4* __restrict__ txy, const int2* __restrict__ kxy,
    const float2* __restrict__ cs, const ZParam* __restrict__ zp, unsigned nview, unsigned m0, unsigned mc,
    const __grid_constant__ CUtensorMap vals, unsigned view_rows, float* __restrict__ vol,
    const float* __restrict__ sens, unsigned long long* __restrict__ npairs, unsigned* give_up)
{
    constexpr unsigned kPair = 2 * sizeof(ST);  // bytes of a pair
    constexpr int NE = 8 * PS * 32;  // epilogue entries per warp
    constexpr int VB = kStageBytes / (4 * RB);  // base views per stage
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ unsigned long long full[kStages], empty[kStages];
    __shared__ int stage_u[kStages * VB], first_u[32];
    __shared__ StagedItem items[kStagedWarps][32];
    unsigned char* const smem0 = smem + ((128u - (smem_addr(smem) & 127u)) & 127u);
    float4* const szq = reinterpret_cast<float4*>(smem0);  // z planes of the staged rows, as in bp_gather_kernel
    unsigned char* const stage0 = smem0 + (((size_t)S.rows * sizeof(float4) + 127) & ~(size_t)127);
    float* const epi = reinterpret_cast<float*>(stage0);
    const unsigned zq = smem_addr(szq), sq = smem_addr(stage0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int H = G.X / 2;
    const int i0 = blockIdx.x * kStagedTX, j0 = blockIdx.y * kStagedTY;
    const int i = i0 + warp % kStagedTX, j = j0 + (warp / kStagedTX) % kStagedTY;
    const bool active = warp < kStagedWarps && i < H && j < H;
    const unsigned nactive = (unsigned)(min(kStagedTX, H - i0) * min(kStagedTY, H - j0));
    const unsigned Q = nview / 4u;
    const unsigned nitem = SET ? 4u * mc : nview;
    auto view_of = [&](unsigned it) { return SET ? m0 + it % mc + (it / mc) * Q : it; };
    if (threadIdx.x == 0) {
        for (unsigned s = 0; s < kStages; ++s) {
            mbar_init(smem_addr(&full[s]), 1u);
            mbar_init(smem_addr(&empty[s]), nactive);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const float Tx0 = G.P0[0] + i0 * G.vox[0], Tx1 = Tx0 + kStagedTX * G.vox[0];
    const float Ty0 = G.P0[1] + j0 * G.vox[1], Ty1 = Ty0 + kStagedTY * G.vox[1];
    const float Xa = G.P0[0] + i * G.vox[0], Xb = Xa + G.vox[0];
    const float Ya = G.P0[1] + j * G.vox[1], Yb = Ya + G.vox[1];
    const float rx = fmaxf(fabsf(Tx0), fabsf(Tx1)), ry = fmaxf(fabsf(Ty0), fabsf(Ty1));
    const float rad = sqrtf(rx * rx + ry * ry) * 1.0001f;  // the tile's columns lie within it at every view
    const float dz32 = 32.0f * G.vox[2];
    const int Zh = G.Z / 2;
    const int Nh = G.Nv / 2;
    const unsigned nuse = (nitem + VB - 1) / VB;  // stage uses per chunk
    unsigned base = 0;                            // and before this chunk
    bool ok = true;
    // A chunk's sums are taken with every product added, a row without a positive length
    // as 0 * value.  Where a sum comes out not finite -- a value was not -- the chunk is
    // taken again (exact) with only the products of positive lengths, which gives a value
    // to the voxels that its ray crosses and to no others.
    bool exact = EPI == 2;
    for (int k0 = 0; k0 < Zh; base += nuse) {
        // the rows that this chunk's lower voxels can meet, and their z planes
        float flo, fhi;
        staged_rows(C, G.P0[2] + (float)k0 * G.vox[2], G.P0[2] + (float)min(k0 + 32 * PS, Zh) * G.vox[2], G.Rf - rad,
                    G.Rf + rad, flo, fhi);
        const int p0 = min(max(0, (int)floorf(flo)), Nh) & ~3;
        const int nrow = min(((min(Nh, max((int)ceilf(fhi), p0)) - p0 + 1) + 3) & ~3, S.rows);
        __syncthreads();  // barriers set up; the last chunk's epilogue is done
        for (int q = threadIdx.x; q < nrow; q += blockDim.x) {
            const ZParam z = zp[min(p0 + q, G.Nv - 1)];
            const float kc = (float)z.kc;
            szq[q] = (z.S > 0.0f) ? make_float4(z.S, z.O, kc, kc - 1.0f) : make_float4(z.S, z.O, kc - 1.0f, kc);
        }
        if (k0 > 0) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        float2 acc[4][PS];  // {lower voxel, its mirror} in the four columns
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int s = 0; s < PS; ++s) acc[r][s] = make_float2(0.0f, 0.0f);
        const int nslot = min(PS, max(0, (Zh - k0 - lane + 31) / 32));
        if (warp == kStagedWarps) {
            // the loading warp: VB items' detector columns into each stage, in turn
            const unsigned bytes = 4u * (unsigned)(S.rows * S.cols) * kPair;
            unsigned st = base % kStages, ph = (base / kStages) & 1u;
            for (unsigned n = 0; n < nuse && ok; ++n) {
                const unsigned i0 = n * VB, cnt = min((unsigned)VB, nitem - i0);
                if (i0 % 32u == 0u) {  // 32 items' first detector columns, one per lane
                    __syncwarp();
                    if (i0 + lane < nitem)
                        first_u[lane] = staged_first_column(G, C, __ldg(cs + view_of(i0 + lane)), Tx0, Tx1, Ty0, Ty1);
                    __syncwarp();
                }
                ok = mbar_wait(smem_addr(&empty[st]), ph ^ 1u);
                const unsigned bar = smem_addr(&full[st]);
                if (ok && lane < VB) stage_u[st * VB + lane] = first_u[(i0 + lane) % 32u];
                __syncwarp();
                if (ok && lane == 0) {
                    mbar_expect(bar, bytes * cnt);
                    for (unsigned b = 0; b < cnt; ++b) {
                        const int u = first_u[(i0 + b) % 32u];
                        unsigned w = view_of(i0 + b);
#pragma unroll
                        for (int r = 0; r < 4; ++r) {
                            tile_load(sq + st * kStageBytes + (b * 4 + r) * RB, &vals, p0, (int)(w * view_rows) + u, bar);
                            w = (w + Q >= nview) ? w + Q - nview : w + Q;
                        }
                    }
                }
                if (!ok) {  // a warp does not answer: let the copies in flight land, then stop
                    if (lane == 0) report_give_up(give_up);
                    for (unsigned b = 1; b <= min(n, kStages); ++b) {
                        const unsigned use = base + n - b;
                        mbar_wait(smem_addr(&full[use % kStages]), (use / kStages) & 1u);
                    }
                }
                if (++st == kStages) {
                    st = 0;
                    ph ^= 1u;
                }
            }
        } else if (active) {
            const float fk0 = (float)(k0 + lane);
            const float zl0 = fmaf(fk0, G.vox[2], G.P0[2]), zh0 = zl0 + G.vox[2];
            // rows relative to p0, with bp_gather_kernel's margins
            const float oz_lo = C.oz - 0.002f - (float)p0, oz_hi = C.oz + 0.002f - (float)p0;
            const unsigned last = (unsigned)nrow - 1u, colb = (unsigned)S.rows * kPair;
            // row a of the staged rows: its length through lower voxel s of this lane, times
            // its pairs in the four views (RB bytes apart from col)
            auto add_row = [&](auto exact_tag, int s, float A, float B, unsigned a, unsigned col) {
                const float4 zr = lds_planes(zq + a * 16u);
                const float t = fk0 + (float)(32 * s);
                const float lo = fmaf(t - zr.z, zr.x, zr.y), hi = fmaf(t - zr.w, zr.x, zr.y);
                const float L = fminf(B, hi) - fmaxf(A, lo);
                const unsigned x = col + a * kPair;
                if constexpr (decltype(exact_tag)::value) {
                    if (!(L > 0.0f)) return;
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const auto p = lds_pair(x + r * RB, ST());
                        acc[r][s].x = (EPI == 2) ? acc[r][s].x + 1.0f : fmaf(L, widen_lo(p), acc[r][s].x);
                        acc[r][s].y = (EPI == 2) ? acc[r][s].y + 1.0f : fmaf(L, widen_hi(p), acc[r][s].y);
                    }
                } else {
                    const float Lp = fmaxf(L, 0.0f);
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const auto p = lds_pair(x + r * RB, ST());
                        fma_pair(acc[r][s], Lp, make_float2(widen_lo(p), widen_hi(p)));
                    }
                }
            };
            // one detector column, several candidate rows per voxel or exact sums: col = the
            // first view's pairs of it
            auto rows_general = [&](auto exact_tag, const StagedItem& I, unsigned col) {
                const float P0a = fmaf(zl0, I.ca, oz_lo), P0b = fmaf(zl0, I.cb, oz_lo);
                const float P1a = fmaf(zh0, I.ca, oz_hi), P1b = fmaf(zh0, I.cb, oz_hi);
                unsigned a[PS];
                int more = 0;  // further candidate rows of this lane's voxels, at most
#pragma unroll
                for (int s = 0; s < PS; ++s) {
                    const float f0 = fminf(fmaf((float)s, I.pa, P0a), fmaf((float)s, I.pb, P0b));
                    const float f1 = fmaxf(fmaf((float)s, I.pa, P1a), fmaf((float)s, I.pb, P1b));
                    a[s] = min(__float2uint_ru(f0), last);
                    more = max(more, min(__float2int_rd(f1), (int)last) - (int)a[s]);
                }
                more = __reduce_max_sync(0xffffffffu, more);
                for (int n = 0; n <= more; ++n)
#pragma unroll
                    for (int s = 0; s < PS; ++s)
                        if (n == 0 || a[s] + (unsigned)n <= last) add_row(exact_tag, s, I.A, I.B, a[s] + (unsigned)n, col);
            };
            const int wshift = __ffs(S.wide) - 1;
            const int per = 32 / S.wide;  // views whose items a warp sets up at a time
            unsigned st = base % kStages, ph = (base / kStages) & 1u;
            for (unsigned vb = 0; vb < nitem; vb += per) {
                const unsigned nb = min((unsigned)per, nitem - vb);
                bool valid = false;
                {
                    const unsigned q = (unsigned)(lane / S.wide);
                    StagedItem it;
                    if (q < nb) {
                        const unsigned m = view_of(vb + q);
                        valid = staged_item(G, C, txy, kxy, __ldg(cs + m), m, lane % S.wide, i, j, Xa, Xb, Ya, Yb,
                                            oz_hi - oz_lo, dz32, it);
                        if (exact) it.one = 0;
                        if (valid) items[warp][lane] = it;
                    }
                }
                unsigned mask = __ballot_sync(0xffffffffu, valid);
                __syncwarp();
                for (unsigned q = 0; q < nb; q += VB) {
                    // the stage's items: bits q wide .. (q + VB) wide - 1 of the mask
                    unsigned mine = (S.wide * VB >= 32) ? mask : (mask >> (q * S.wide)) & ((1u << (S.wide * VB)) - 1u);
                    if (ok) ok = mbar_wait(smem_addr(&full[st]), ph);
                    for (; mine != 0u; mine &= mine - 1u) {
                        const unsigned e = (unsigned)__ffs(mine) - 1u, b = e >> wshift;
                        const StagedItem I = items[warp][q * S.wide + e];
                        const unsigned col = sq + st * kStageBytes + b * (4 * RB) +
                                             (unsigned)min(max(I.u - stage_u[st * VB + b], 0), S.cols - 1) * colb;
                        if (I.one) {  // one candidate row per voxel, clamped to a staged row
                            const float P0a = fmaf(zl0, I.ca, oz_lo);
#pragma unroll
                            for (int s = 0; s < PS; ++s)
                                add_row(std::false_type{}, s, I.A, I.B,
                                        min(__float2uint_ru(fmaf((float)s, I.pa, P0a)), last), col);
                        } else if (exact) {
                            rows_general(std::true_type{}, I, col);
                        } else {
                            rows_general(std::false_type{}, I, col);
                        }
                    }
                    __syncwarp();  // the stage is read
                    if (lane == 0) mbar_arrive(smem_addr(&empty[st]));
                    if (++st == kStages) {
                        st = 0;
                        ph ^= 1u;
                    }
                }
                __syncwarp();  // the next batch rewrites the items
            }
            if (!ok) {  // a stage never came: the sums are not the answer
                if (lane == 0) report_give_up(give_up);
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int s = 0; s < PS; ++s) acc[r][s].x = acc[r][s].y = __int_as_float(0x7fffffff);
            }
        }
        if (EPI != 2) {
            bool bad = false;
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int s = 0; s < PS; ++s) bad |= s < nslot && !(isfinite(acc[r][s].x) && isfinite(acc[r][s].y));
            if (__syncthreads_or(bad && ok && !exact)) {
                exact = true;
                continue;
            }
            exact = false;
        }
        if (EPI == 2) {  // pair counts of the four columns
            unsigned long long c = 0;
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int s = 0; s < PS; ++s)
                    if (s < nslot) c += (unsigned long long)acc[r][s].x + (unsigned long long)acc[r][s].y;
            for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
            if (lane == 0 && c) atomicAdd(npairs, c);
            k0 += 32 * PS;
            continue;
        }
        // every stage is read (the barrier above): its memory takes the sums
        if (warp < kStagedWarps) {
            float* const o = epi + warp * NE;
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int s = 0; s < PS; ++s) {
                    o[((r * 2) * PS + s) * 32 + lane] = acc[r][s].x;
                    o[((r * 2 + 1) * PS + s) * 32 + lane] = acc[r][s].y;
                }
        }
        __syncthreads();
        // one voxel per thread, the tile's columns fastest (x neighbours adjacent)
        const size_t plane = (size_t)G.X * G.Y;
        for (int q = threadIdx.x; q < kStagedWarps * NE; q += blockDim.x) {
            const int w = q % kStagedWarps, e = q / kStagedWarps;
            const int r = e / (2 * PS * 32), h = (e / (PS * 32)) & 1, k = k0 + e % (PS * 32);
            // columns d_1 and d_3 run along x with the base column's y
            const int wi = (r & 1) ? w / kStagedTX : w % kStagedTX, wj = (r & 1) ? w % kStagedTX : w / kStagedTX;
            const int bi = i0 + wi, bj = j0 + wj;
            if (bi >= H || bj >= H || k >= Zh) continue;
            const int x = (r == 0) ? bi : (r == 1) ? bj : (r == 2) ? G.X - 1 - bi : G.X - 1 - bj;
            const int y = (r == 0) ? bj : (r == 1) ? G.X - 1 - bi : (r == 2) ? G.X - 1 - bj : bi;
            const int z = h ? G.Z - 1 - k : k;
            const size_t v = (size_t)z * plane + (size_t)y * G.X + (size_t)x;
            const float hv = epi[(wj * kStagedTX + wi) * NE + e];
            vol[v] = (EPI == 1) ? gather_update(vol[v], hv, sens[v]) : hv;
        }
        k0 += 32 * PS;
    }
}

// A wait on a barrier that nothing arrives at, with a limit of about ten milliseconds.
__global__ void wait_selftest_kernel(unsigned* give_up)
{
    __shared__ unsigned long long bar;
    mbar_init(smem_addr(&bar), 1u);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (!mbar_wait(smem_addr(&bar), 0u, 20000000ll)) report_give_up(give_up);
}

}  // namespace exact

// ---- host side -----------------------------------------------------------------------------

recon_status_t launch_wait_selftest(Plan& P, cudaStream_t s)
{
    exact::wait_selftest_kernel<<<1, 1, 0, s>>>(P.d_give_up);
    RB_CUDA(cudaGetLastError());
    return RECON_OK;
}

// Detector columns whose rays can meet a rectangle of diagonal d mm anywhere in the
// volume: its shadow is at most d * |Ry| / depth * sqrt(1 + tan^2) / du pitches wide.
static int staged_span(const Plan& P, double d, double rad)
{
    const ExactGeom& E = P.eg;
    const double dmin = (double)E.Rf - rad, tan = rad / dmin;
    return (int)std::floor(d / dmin * std::sqrt(1.0 + tan * tan) * std::fabs((double)E.Ry / E.du) + 0.05) + 1;
}

// staged_item finds its detector columns and row coefficients with quick divisions, good to
// two units in the last place (exact ones made the MLEM iteration at 256^3 1.2 % slower, the
// one at 512^3 1.4 %).  What they may miss stays inside the margins, 0.01 column and 0.002
// row, on detectors of these sizes.  Rows: a bound z * ez / depth lies up to Nv / 2 from the
// centre with a relative error of 4 (division) + 5 (its operands and coefficients) times
// 2^-24, and is rounded twice more at up to Nv: 0.0016 row at 4096.  Columns: 14 times 2^-24
// of up to Nu, 0.007 column at 8192.  (Exact division would give 0.0012 and 0.005.)
static bool staged_bounds_hold(const Plan& P) { return P.eg.Nv <= 4096 && P.eg.Nu <= 8192; }

// Voxels meet clearly more than one detector row per detector column and view: the rows'
// distance and the slant of a voxel column's piece, where both are largest.
bool several_candidate_rows(const Plan& P)
{
    const ExactGeom& E = P.eg;
    const double vx = E.vox[0], vy = E.vox[1], vz = E.vox[2], ez = std::fabs((double)E.Ry / E.dv);
    const double near = (double)E.Rf - 0.5 * std::hypot(E.X * vx, E.Y * vy);
    return !(near > 0.0) || (vz + 0.5 * E.Z * vz * std::hypot(vx, vy) / near) * ez / near > 1.05;
}

// Most detector columns that one voxel column meets in a view, or 0 where staged_item does
// not serve: its bounds do not hold, or the volume comes near the source (where a piece
// could lie behind it).
int staged_wide(const Plan& P)
{
    const ExactGeom& E = P.eg;
    if (!staged_bounds_hold(P)) return 0;
    const double vx = E.vox[0], vy = E.vox[1];
    const double rad = std::hypot(0.5 * E.X * vx + 32 * vx, 0.5 * E.Y * vy + 4 * vy) * 1.001;
    return rad < 0.9 * (double)E.Rf ? staged_span(P, std::hypot(vx, vy), rad) : 0;
}

// The boxes that tiles read in chunks of 32 * slots slices of the lower half, of detector
// columns in row pairs 0 .. Nv/2 (in multiples of four pairs): S->wide, cols and rows.
// False where no staged gather serves: a detector too large for staged_item's bounds, a
// volume that comes near the source (a piece could then lie behind it), a voxel column that
// meets more than eight detector columns, or a box of more than 256 a side.
static bool staged_boxes(const Plan& P, int slots, exact::StagedShape* S)
{
    const ExactGeom& E = P.eg;
    if (!staged_bounds_hold(P)) return false;
    const double vx = E.vox[0], vy = E.vox[1], vz = E.vox[2];
    const double tx = exact::kStagedTX * vx, ty = exact::kStagedTY * vy;
    const double rad = std::hypot(0.5 * E.X * vx + tx, 0.5 * E.Y * vy + ty) * 1.001;
    if (!(rad < 0.9 * (double)E.Rf)) return false;
    const double ez = (double)E.Ry / E.dv, oz = -((double)E.Dz + E.vd0) / E.dv;
    const int wide = staged_span(P, std::hypot(vx, vy), rad);
    if (wide > 8) return false;
    S->wide = wide <= 1 ? 1 : wide <= 2 ? 2 : wide <= 4 ? 4 : 8;
    S->cols = staged_span(P, std::hypot(tx, ty), rad);
    constexpr int align = 4;
    const int Zs = E.Z / 2, top = E.Nv / 2;
    int rows = align;
    for (int k0 = 0; k0 < Zs; k0 += 32 * slots) {
        const double zb = E.P0[2] + k0 * vz, zt = E.P0[2] + std::min(k0 + 32 * slots, Zs) * vz;
        const double dn = E.Rf - rad, df = E.Rf + rad;
        const double lo = std::min(zb / dn * ez, zb / df * ez) + oz - 2.0;
        const double hi = std::max(zt / dn * ez, zt / df * ez) + oz + 2.0;
        if (!(lo > -1e8 && hi < 1e8)) return false;
        const int a = std::min(std::max(0, (int)std::floor(lo)), top) / align * align;
        const int b = std::max(a, std::min(top, (int)std::ceil(hi)));
        rows = std::max(rows, (b - a + align) / align * align);
    }
    S->rows = rows;
    return S->rows <= 256 && S->cols <= 256;
}

// The quarter-turn kernel's stages for chunks of 32 * slots slices of the lower half, or
// false where bp_gather_quarter_kernel is the quarter-turn gather instead: no boxes, or
// boxes of more than 12 KiB (a detector several times finer than the voxels: its rows and
// columns then outgrow the two stages that a block's shared memory holds).
static bool staged_shape(const Plan& P, int slots, size_t value_bytes, exact::StagedShape* out, int* region,
                         size_t* smem)
{
    exact::StagedShape S{};
    if (!staged_boxes(P, slots, &S)) return false;
    const size_t used = (size_t)S.cols * S.rows * 2 * value_bytes;
    if (used > 12288) return false;
    *region = used <= 6144 ? 6144 : 12288;
    const size_t planes = ((size_t)S.rows * sizeof(float4) + 127) / 128 * 128;
    const size_t epilogue = sizeof(float) * exact::kStagedWarps * 8 * slots * 32;
    const size_t room = kStagedSmem - planes;
    const size_t stages = (size_t)exact::kStages * exact::kStageBytes;
    if (stages > room || epilogue > room) return false;
    *out = S;
    *smem = 128 + planes + std::max(stages, epilogue);  // 128: the base's alignment
    return true;
}

// The driver's tensor map encoder, looked up once.
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder()
{
    static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }();
    return fn;
}

// A table of `table_rows` detector columns of `pitch` row pairs (moved as one element of
// `pair` bytes), read in boxes of S.rows pairs x S.cols detector columns.
static bool column_map(const exact::StagedShape& S, const void* vals, size_t pitch, size_t pair, size_t table_rows,
                       CUtensorMap* map)
{
    const auto encode = tensor_map_encoder();
    if (!encode || reinterpret_cast<uintptr_t>(vals) % 16 != 0 || pitch * pair % 16 != 0) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)pitch, (cuuint64_t)table_rows};
    const cuuint64_t strides[1] = {(cuuint64_t)(pitch * pair)};
    const cuuint32_t box[2] = {(cuuint32_t)S.rows, (cuuint32_t)S.cols}, step[2] = {1, 1};
    const CUtensorMapDataType type = pair == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_UINT32;
    return encode(map, type, 2, const_cast<void*>(vals), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int EPI, class ST, int PS, int RB, bool SET>
static recon_status_t launch_staged(Plan& P, const exact::StagedShape& S, size_t smem, const CUtensorMap& map,
                                    unsigned view_rows, float* vol, const float* sens, cudaStream_t s,
                                    unsigned long long* npairs, unsigned m0, unsigned mc)
{
    const ExactGeom& E = P.eg;
    auto kernel = exact::bp_staged_quarter_kernel<EPI, ST, PS, RB, SET>;
    RB_CHECK(allow_dynamic_smem(kernel, 128 + kStagedSmem));
    note_kernel(RECON_PROJECTOR_BACK, "bp_staged_quarter_kernel");
    const int H = E.X / 2;
    const dim3 grid((H + exact::kStagedTX - 1) / exact::kStagedTX, (H + exact::kStagedTY - 1) / exact::kStagedTY);
    kernel<<<grid, exact::kStagedThreads, smem, s>>>(E, gather_const(P, vol, sens), S, P.d_txy, P.d_kxy, P.d_cs, P.d_zp,
                                                     P.nviews, m0, mc, map, view_rows, vol, sens, npairs, P.d_give_up);
    RB_CUDA(cudaGetLastError());
    return RECON_OK;
}

// Voxel pairs per lane: the lower half's height in as few chunks of at most 4 x 32
// slices as possible, split evenly.
static int staged_slots(int Z)
{
    const int half = Z / 2, chunks = (half + 127) / 128;
    return std::min(4, std::max(1, (half + 32 * chunks - 1) / (32 * chunks)));
}

// The quarter-turn gather over base views m0 .. m0 + mc - 1 of each quarter (set), or
// all views; *served = false (and nothing launched) where its stages do not fit.
template <int EPI, class ST>
recon_status_t staged_quarter_gather(Plan& P, const ST* vals, size_t view_stride, float* vol, const float* sens,
                                     cudaStream_t s, unsigned long long* npairs, bool set, unsigned m0, unsigned mc,
                                     bool* served)
{
    exact::StagedShape S;
    size_t smem = 0;
    int region = 0;
    const int slots = staged_slots(P.eg.Z);
    CUtensorMap map;
    // view_stride 0: the same table for every view (the weights of the sensitivity)
    const unsigned view_rows = view_stride ? (unsigned)P.eg.Nu : 0u;
    const size_t table_rows = view_stride ? (size_t)P.eg.Nu * P.nviews : (size_t)P.eg.Nu;
    // Fewer tiles than half the SMs: bp_gather_quarter_kernel, whose tiles are half as large, is
    // as fast or faster at the weights (one table for every view: 64 x 64 x 300, 80 views, 88
    // against 92 us, 64 x 64 x 512 103 / 113) and, where voxels have several candidate rows, at
    // volumes of two chunks (48 x 48 x 300 293 / 305, 64 x 64 x 512 424 / 451).
    const int H = P.eg.X / 2, tiles = (H + exact::kStagedTX - 1) / exact::kStagedTX * ((H + exact::kStagedTY - 1) / exact::kStagedTY);
    const bool few_tiles = 2 * tiles <= P.sm_count &&
                           (EPI == 0 && view_stride == 0 ? P.eg.Z > 128 : P.eg.Z > 256 && several_candidate_rows(P));
    *served = P.d_give_up && !few_tiles && table_rows < 0x7fffffff && staged_shape(P, slots, sizeof(ST), &S, &region, &smem) &&
              column_map(S, vals, pair_entries(P.eg.Nv), 2 * sizeof(ST), table_rows, &map);
    if (!*served) return RECON_OK;
    auto run = [&](auto ps) -> recon_status_t {
        constexpr int PS = decltype(ps)::value;
        auto go = [&](auto rb) -> recon_status_t {
            constexpr int RB = decltype(rb)::value;
            if constexpr (EPI == 0) {
                if (set)
                    return launch_staged<EPI, ST, PS, RB, true>(P, S, smem, map, view_rows, vol, sens, s, npairs, m0, mc);
            }
            return launch_staged<EPI, ST, PS, RB, false>(P, S, smem, map, view_rows, vol, sens, s, npairs, m0, mc);
        };
        return region == 6144 ? go(std::integral_constant<int, 6144>{}) : go(std::integral_constant<int, 12288>{});
    };
    switch (slots) {
        case 1: return run(std::integral_constant<int, 1>{});
        case 2: return run(std::integral_constant<int, 2>{});
        case 3: return run(std::integral_constant<int, 3>{});
        default: return run(std::integral_constant<int, 4>{});
    }
}

#define RB_STAGED(EPI, ST)                                                                                          \
    template recon_status_t staged_quarter_gather<EPI, ST>(Plan&, const ST*, size_t, float*, const float*,          \
                                                           cudaStream_t, unsigned long long*, bool, unsigned, unsigned, \
                                                           bool*);
RB_STAGED(0, float)
RB_STAGED(1, float)
RB_STAGED(2, float)
RB_STAGED(0, __nv_bfloat16)
RB_STAGED(1, __nv_bfloat16)
#undef RB_STAGED

}  // namespace rb
