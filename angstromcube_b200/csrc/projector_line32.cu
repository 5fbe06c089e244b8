// FP32 instantiations of the projector kernels along lines of cubes (projector_line.cuh).
#include "projector_line.cuh"

namespace a43g {

bool prepare_line_kernels32() { return line::prepare<float>(); }

bool launch_project_line(DevicePlan &dp, float *apc, float const *x, void const *tab, LineScratch const &sc,
                         cudaStream_t st) {
    return line::launch_project<float>(dp, apc, x, tab, sc, st);
}

bool launch_add_line(DevicePlan &dp, float *y, float const *cad, uint16_t const *colIndex, cudaStream_t st) {
    return line::launch_add<float>(dp, y, cad, colIndex, dp.line_tab32.ptr, st);
}

} // namespace a43g
