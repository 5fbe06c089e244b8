// FP64 instantiations of the projector kernels along lines of cubes (projector_line.cuh).
#include "projector_line.cuh"

namespace a43g {

bool prepare_line_kernels64() { return line::prepare<double>(); }

bool launch_project_line(DevicePlan &dp, double *apc, double const *x, void const *tab, LineScratch const &sc,
                         cudaStream_t st) {
    return line::launch_project<double>(dp, apc, x, tab, sc, st);
}

bool launch_add_line(DevicePlan &dp, double *y, double const *cad, uint16_t const *colIndex, cudaStream_t st) {
    return line::launch_add<double>(dp, y, cad, colIndex, dp.line_tab64.ptr, st);
}

} // namespace a43g
