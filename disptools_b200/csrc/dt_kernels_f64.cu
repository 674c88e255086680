// FP64 instantiation of the stencil kernels.  This file is compiled with
// -fmad=false: no multiply-add contraction, so every per-voxel expression
// rounds exactly as the reference C library computes it.
#include "dt_jacobian.cuh"
#include "dt_kernels_tma.cuh"

namespace dtb {
DTB_INSTANTIATE(double)
DTB_INSTANTIATE_TMA(double)
DTB_INSTANTIATE_JACOBIAN(double)
// The logs of a map in FP64, of fields of either type.
template cudaError_t launch_log_jacobian<float>(const float *, const Geom &, double *, double, bool, bool, double, int,
                                                cudaStream_t);
template cudaError_t launch_log_jacobian<double>(const double *, const Geom &, double *, double, bool, bool, double,
                                                 int, cudaStream_t);
}
