// Plane transform kernels, FP64, grids from 72 (one plane pair fits up to 108) (pgj_planes.cuh).
#include "pgj_planes.cuh"

namespace pgj {
void planes_f64c(PlaneKernels* out, int* count) {
  out[(*count)++] = planes_entry<PlaneCfg<72, double>>();
  out[(*count)++] = planes_entry<PlaneCfg<80, double>>();
  out[(*count)++] = planes_entry<PlaneCfg<90, double>>();
  out[(*count)++] = planes_entry<PlaneCfg<96, double>>();
  out[(*count)++] = planes_entry<PlaneCfg<100, double>>();
  out[(*count)++] = planes_entry<PlaneCfg<108, double>>();
}
}  // namespace pgj
