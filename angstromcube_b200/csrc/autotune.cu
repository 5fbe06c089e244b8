// Autotuner of the action's schedule for one plan on the current device.
//
// The kernels have a few schedule parameters whose best value depends on the plan (how many
// blocks, how many atom images per block, how long the z-lines are) and on the GPU:
//   * prj_chunk   : blocks of one (image, source) list per projection CTA (the cubes-per-CTA
//                   schedule of the projection: longer chunks amortize the start and the
//                   partial sums, shorter ones balance the load)   {12, 24, 40}
//   * use_tc      : FP32 projector on the tensor cores (3xTF32) or on the CUDA cores
// Each parameter is tuned in turn (coordinate descent), every candidate timed with CUDA events
// on the caller's stream: two untimed applications, then the mean of three.  Scratch vectors
// for x and y are allocated for the duration of the call.
#include "device.cuh"

#include <cstdio>
#include <string>
#include <vector>

namespace a43g {

namespace {

template <typename T>
bool time_part(DevicePlan &dp, int part, T *y, T const *x, uint16_t const *ci, cudaStream_t st, float &ms) {
    cudaEvent_t e0, e1;
    A43G_CUDA_TRY(cudaEventCreate(&e0));
    A43G_CUDA_TRY(cudaEventCreate(&e1));
    auto run = [&]() {
        return (0 == part) ? launch_local<T>(dp, y, x, st) : launch_dyadic<T>(dp, y, x, ci, st);
    };
    bool ok = run() && run();
    if (ok) {
        cudaEventRecord(e0, st);
        for (int r = 0; r < 3 && ok; ++r) ok = run();
        cudaEventRecord(e1, st);
        ok = ok && cudaSuccess == cudaEventSynchronize(e1);
        cudaEventElapsedTime(&ms, e0, e1);
        ms /= 3;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return ok;
}

} // namespace

template <typename T>
bool autotune(GreenPlan const &hp, DevicePlan &dp, cudaStream_t st, std::string &report) {
    size_t const n = size_t(dp.nnzb)*8192;
    if (0 == n) return true;
    if (!readers_done(st)) return false;            // the work items are replaced below
    DeviceBuffer bx, by;
    if (!bx.alloc(n*sizeof(T)) || !by.alloc(n*sizeof(T))) return false;
    A43G_CUDA_TRY(cudaMemsetAsync(bx.ptr, 0x3c, n*sizeof(T), st));   // finite values of moderate size
    T *y = dptr<T>(by);
    T const *x = dptr<T>(bx);
    uint16_t const *ci = dptr<uint16_t>(dp.colindx);
    char line[160];
    float ms = 0;
    if (dp.nAI > 0 && dp.nCols > 0) {
        uint32_t best = dp.prj_chunk; float tbest = 1e30f;
        for (uint32_t c : {12u, 24u, 40u}) {
            dp.prj_chunk = c;
            if (!build_prj_items(hp, dp) || !time_part<T>(dp, 1, y, x, ci, st, ms)) return false;
            std::snprintf(line, sizeof(line), "projector chunk %2u blocks: %.3f ms\n", c, ms); report += line;
            if (ms < tbest) { tbest = ms; best = c; }
        }
        dp.prj_chunk = best;
        if (!build_prj_items(hp, dp)) return false;
        if (sizeof(T) == 4) {
            if (tc_projector_supported(dp)) {
                bool const before = dp.use_tc;
                float t[2] = {0, 0};
                for (int tc = 0; tc < 2; ++tc) {
                    dp.use_tc = (1 == tc);
                    if (!time_part<T>(dp, 1, y, x, ci, st, t[tc])) { dp.use_tc = before; return false; }
                    std::snprintf(line, sizeof(line), "projector on the %s: %.3f ms\n", tc ? "tensor cores" : "CUDA cores", t[tc]);
                    report += line;
                }
                dp.use_tc = t[1] < t[0];
                if (dp.use_tc) {   // a tensor-core run that recorded a wait timeout is not usable
                    int flag = 0;
                    A43G_CUDA_TRY(cudaMemcpyAsync(&flag, dp.dev_error.ptr, sizeof(int), cudaMemcpyDeviceToHost, st));
                    A43G_CUDA_TRY(cudaStreamSynchronize(st));
                    if (flag) dp.use_tc = false;
                }
            }
        }
    }
    std::snprintf(line, sizeof(line), "chosen: projector chunk %u, local %s, %s projector\n",
                  dp.prj_chunk, dp.local_rows ? "plain rows" : "pencils", dp.use_tc ? "tensor-core" : "CUDA-core");
    report += line;
    A43G_CUDA_TRY(cudaStreamSynchronize(st));
    return true;
}

template bool autotune<float>(GreenPlan const &, DevicePlan &, cudaStream_t, std::string &);
template bool autotune<double>(GreenPlan const &, DevicePlan &, cudaStream_t, std::string &);

} // namespace a43g
