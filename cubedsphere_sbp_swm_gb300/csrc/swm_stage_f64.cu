// swm_stage_f64.cu -- double instantiation of the FP64 stage kernels.
#include "swm_launch.h"
#include "swm_stage.cuh"

namespace swm {

// The FP64 stage has no work units; its contexts report one width.
constexpr int kReportedWidth = 64;

cudaError_t launch_derive64(const InstDev<double>& one, const InstDev<double>* many, int ninst,
                            int max_n, cudaStream_t st) {
  return launch_point_derive<double>(one, many, ninst, max_n, st);
}

cudaError_t launch_stage64(int order, const InstDev<double>& one, const InstDev<double>* many,
                           int ninst, int max_n, const Topology& tp, int mode, cudaStream_t st) {
  switch (order) {
    case 21: return launch_point_stage_ord<double, 21>(one, many, ninst, max_n, tp, mode, st);
    case 42: return launch_point_stage_ord<double, 42>(one, many, ninst, max_n, tp, mode, st);
    case 43: return launch_point_stage_ord<double, 43>(one, many, ninst, max_n, tp, mode, st);
    case 63: return launch_point_stage_ord<double, 63>(one, many, ninst, max_n, tp, mode, st);
    default: return cudaErrorInvalidValue;
  }
}

template <>
cudaError_t prepare_stage<double>(int order, StageShape* shape) {
  (void)order;
  shape->ctas_per_sm = 1;
  shape->cols = kReportedWidth;
  shape->tma = 0;
  shape->boxw = shape->rps = shape->nf = 0;
  shape->fixbw = 0;
  return cudaSuccess;
}

template <>
int stage_boxw_max<double>(int cols) {
  (void)cols;
  return 0;
}

template <>
int stage_occupancy<double>(int order, int boxw, int cols, bool fixbw) {
  (void)order;
  (void)boxw;
  (void)cols;
  (void)fixbw;
  return 1;
}

}  // namespace swm
