// Two host threads, each with a plan and a stream of its own, whose plans run the same
// kernels with different amounts of shared memory: no call may fail.
// argv[1]: calls per thread and kind.  Prints one line per kind; exit status 1 on any failure.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <string>
#include <thread>

#include "recon_b200.h"

static recon_geometry_t geometry(unsigned x, unsigned y, unsigned z, float vxy, float vz, unsigned nu, unsigned nv,
                                 float pu, float pv, unsigned views)
{
    recon_geometry_t g{};
    g.cal.R = g.cal.Ry = 800.0f;
    g.cal.Rf = 500.0f;
    g.cal.M = 1.0f;
    g.det.NumAxPixels = nu;
    g.det.NumTAxPixels = nv;
    g.det.AxPixDimMm = pu;
    g.det.TAxPixDimMm = pv;
    g.vox.Xdim = x;
    g.vox.Ydim = y;
    g.vox.Zdim = z;
    g.vox.XVoxSize = g.vox.YVoxSize = vxy;
    g.vox.ZVoxSize = vz;
    g.scan.NumProj = views;
    g.scan.DeltaAng = 360.0f / views;
    g.scan.N_iteration = 1;
    return g;
}

struct Kind {
    const char* name;
    recon_geometry_t geom[2];
    int design;   // recon_options_t.siddon_bp
    int forward;  // project forward instead of back
    unsigned count;
};

static bool run(const Kind& K, int calls)
{
    recon_options_t opt;
    recon_default_options(&opt);
    opt.siddon_bp = (recon_siddon_bp_t)K.design;
    recon_plan_t plan[2] = {nullptr, nullptr};
    for (int q = 0; q < 2; ++q)
        if (recon_plan_create(&K.geom[q], &opt, &plan[q]) != RECON_OK) {
            std::printf("%s: %s\n", K.name, recon_last_error());
            return false;
        }
    std::atomic<int> failed{0};
    std::string message[2];
    auto work = [&](int q) {
        const recon_geometry_t& g = K.geom[q];
        const size_t npix = (size_t)g.det.NumAxPixels * g.det.NumTAxPixels * K.count;
        const size_t nvox = (size_t)g.vox.Xdim * g.vox.Ydim * g.vox.Zdim;
        float *sino = nullptr, *vol = nullptr;
        cudaStream_t s = nullptr;
        if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess ||
            cudaMalloc(&sino, npix * sizeof(float)) != cudaSuccess || cudaMalloc(&vol, nvox * sizeof(float)) != cudaSuccess ||
            cudaMemsetAsync(sino, 0, npix * sizeof(float), s) != cudaSuccess ||
            cudaMemsetAsync(vol, 0, nvox * sizeof(float), s) != cudaSuccess) {
            ++failed;
            message[q] = "set-up";
            return;
        }
        for (int n = 0; n < calls; ++n) {
            const recon_status_t st = K.forward ? recon_fp_views(plan[q], vol, 0, K.count, sino, s)
                                                : recon_bp_views(plan[q], sino, 0, K.count, vol, s);
            if (st != RECON_OK) {
                ++failed;
                message[q] = recon_last_error();
            }
            if (n % 256 == 255) cudaStreamSynchronize(s);
        }
        if (cudaStreamSynchronize(s) != cudaSuccess) ++failed;
        cudaFree(sino);
        cudaFree(vol);
        cudaStreamDestroy(s);
    };
    std::thread other(work, 1);
    work(0);
    other.join();
    for (recon_plan_t p : plan) recon_plan_destroy(p);
    std::printf("%s: %d of %d calls failed %s %s\n", K.name, failed.load(), 2 * calls, message[0].c_str(),
                message[1].c_str());
    return failed.load() == 0;
}

int main(int argc, char** argv)
{
    const int calls = argc > 1 ? std::atoi(argv[1]) : 1000;
    const Kind kinds[] = {
        {"a few views",
         {geometry(32, 32, 32, 1, 1, 64, 32, 1.5f, 2.4f, 8), geometry(32, 32, 32, 1, 1, 64, 3000, 1.5f, 0.04f, 8)},
         RECON_SIDDON_BP_GATHER, 0, 1},
        {"quarter turns, staged",
         {geometry(16, 16, 256, 1, 1, 32, 420, 1.5f, 1.5f, 4), geometry(16, 16, 256, 1, 1, 32, 330, 1.5f, 1.7f, 4)},
         RECON_SIDDON_BP_GATHER, 0, 4},
        {"view range, mirrored pairs",
         {geometry(16, 16, 32, 1, 1, 32, 2400, 1.5f, 0.05f, 16), geometry(16, 16, 32, 1, 1, 32, 4000, 1.5f, 0.03f, 16)},
         RECON_SIDDON_BP_GATHER, 0, 7},
        {"quarter turns",
         {geometry(16, 16, 32, 1, 1, 32, 2400, 1.5f, 0.05f, 4), geometry(16, 16, 32, 1, 1, 32, 4000, 1.5f, 0.03f, 4)},
         RECON_SIDDON_BP_GATHER, 0, 4},
        {"long paths, back",
         {geometry(6200, 4, 4, 0.01f, 1, 16, 8, 6, 1, 2), geometry(8000, 4, 4, 0.01f, 1, 16, 8, 6, 1, 2)},
         RECON_SIDDON_BP_RAY, 0, 2},
        {"long paths, forward",
         {geometry(6200, 4, 4, 0.01f, 1, 16, 8, 6, 1, 2), geometry(8000, 4, 4, 0.01f, 1, 16, 8, 6, 1, 2)},
         RECON_SIDDON_BP_RAY, 1, 2},
    };
    bool ok = true;
    for (const Kind& k : kinds) ok = run(k, calls) && ok;
    return ok ? 0 : 1;
}
