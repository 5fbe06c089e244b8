// Autotuner of the action's schedule for one plan on the current device.
//
// The kernels have a few schedule parameters whose best value depends on the plan (how many
// blocks, how many atom images per block) and on the GPU:
//   * prj_chunk   : positions of one (image, source) list per projection CTA (longer chunks amortize
//                   the start and the partial sums, shorter ones balance the load): what the plan's size
//                   gives (prj_chunk_by_size, the untuned value), or 12, 24, 40 where that is faster by
//                   more than the 2 % that such timings differ
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
bool time_dyadic(DevicePlan &dp, T *y, T const *x, uint16_t const *ci, cudaStream_t st, float &ms) {
    cudaEvent_t e0, e1;
    A43G_CUDA_TRY(cudaEventCreate(&e0));
    A43G_CUDA_TRY(cudaEventCreate(&e1));
    auto run = [&]() { return launch_dyadic<T>(dp, y, x, ci, st); };
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
        uint32_t best = 0;                          // 0: by the plan's size
        float tsize = 0, tbest = 0;
        bool const tc_before = dp.use_tc;
        dp.use_tc = false;                          // the tensor-core projection reads no work items
        bool ok = true;
        for (uint32_t c : {0u, 12u, 24u, 40u}) {
            dp.prj_chunk = c;
            ok = build_prj_items(hp, dp) && time_dyadic<T>(dp, y, x, ci, st, ms);
            if (!ok) break;
            std::snprintf(line, sizeof(line), "projector chunk %2u blocks%s: %.3f ms\n", c ? c : prj_chunk_by_size(hp),
                          c ? "" : " (by the plan's size)", ms);
            report += line;
            if (0 == c) tsize = tbest = ms;
            else if (ms < 0.98f*tsize && ms < tbest) { tbest = ms; best = c; }
        }
        dp.use_tc = tc_before;
        dp.prj_chunk = best;
        if (!readers_done(st) || !build_prj_items(hp, dp) || !ok) return false;
        if (sizeof(T) == 4) {
            if (tc_projector_supported(dp)) {
                bool const before = dp.use_tc;
                if (!ensure_tc_tables(hp, dp)) return false;
                float t[2] = {0, 0};
                for (int tc = 0; tc < 2; ++tc) {
                    dp.use_tc = (1 == tc);
                    if (!time_dyadic<T>(dp, y, x, ci, st, t[tc])) { dp.use_tc = before; return false; }
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
                if (!dp.use_tc) dp.slot_H32.release();
            }
        }
    }
    std::snprintf(line, sizeof(line), "chosen: projector chunk %u, local %s, %s projector\n",
                  dp.prj_chunk ? dp.prj_chunk : prj_chunk_by_size(hp), dp.local_rows ? "plain rows" : "pencils",
                  dp.use_tc ? "tensor-core" : "CUDA-core");
    report += line;
    A43G_CUDA_TRY(cudaStreamSynchronize(st));
    return true;
}

template bool autotune<float>(GreenPlan const &, DevicePlan &, cudaStream_t, std::string &);
template bool autotune<double>(GreenPlan const &, DevicePlan &, cudaStream_t, std::string &);

} // namespace a43g
