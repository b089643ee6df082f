// swm_stage_f64.cu -- double instantiation of the FP64 stage kernels.
#include "swm_launch.h"
#include "swm_stage.cuh"

namespace swm {

cudaError_t launch_derive64(const InstDev<double>& one, const PointBatch<double>& b, cudaStream_t st) {
  return launch_point_derive<double>(one, b, st);
}

cudaError_t launch_stage64(int order, const InstDev<double>& one, const PointBatch<double>& b, const Topology& tp,
                           int mode, cudaStream_t st) {
  switch (order) {
    case 21: return launch_point_stage_ord<double, 21>(one, b, tp, mode, st);
    case 42: return launch_point_stage_ord<double, 42>(one, b, tp, mode, st);
    case 43: return launch_point_stage_ord<double, 43>(one, b, tp, mode, st);
    case 63: return launch_point_stage_ord<double, 63>(one, b, tp, mode, st);
    default: return cudaErrorInvalidValue;
  }
}

int stage64_blocks(int order, int n) {
  return (order == 21 ? point_ranges<21>(n) : order == 42 ? point_ranges<42>(n) : order == 43 ? point_ranges<43>(n)
                                                                               : point_ranges<63>(n)).total / PT_TPB;
}

}  // namespace swm
