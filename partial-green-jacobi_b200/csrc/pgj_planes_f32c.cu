// Plane transform kernels, FP32, grids from 72 (pgj_planes.cuh).
#include "pgj_planes.cuh"

namespace pgj {
void planes_f32c(PlaneKernels* out, int* count) {
  out[(*count)++] = planes_entry<PlaneCfg<72, float>>();
  out[(*count)++] = planes_entry<PlaneCfg<80, float>>();
  out[(*count)++] = planes_entry<PlaneCfg<90, float>>();
  out[(*count)++] = planes_entry<PlaneCfg<96, float>>();
  out[(*count)++] = planes_entry<PlaneCfg<100, float>>();
  out[(*count)++] = planes_entry<PlaneCfg<108, float>>();
  out[(*count)++] = planes_entry<PlaneCfg<120, float>>();
  out[(*count)++] = planes_entry<PlaneCfg<128, float>>();
}
}  // namespace pgj
