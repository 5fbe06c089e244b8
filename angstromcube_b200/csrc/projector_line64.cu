// FP64 instantiations of the line-factorized projector (projector_line.cuh).
#include "projector_line.cuh"

namespace a43g {

bool prepare_line_kernels64() { return line::prepare<double>(); }

bool launch_project_line(DevicePlan &dp, double *apc, double const *x, void const *tab, cudaStream_t st) {
    return line::launch_project<double>(dp, apc, x, tab, st);
}

} // namespace a43g
