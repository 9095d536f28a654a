// Plane transform kernels, FP32, grids from 40 to 64 (pgj_planes.cuh).
#include "pgj_planes.cuh"

namespace pgj {
void planes_f32b(PlaneKernels* out, int* count) {
  out[(*count)++] = planes_entry<PlaneCfg<40, float>>();
  out[(*count)++] = planes_entry<PlaneCfg<48, float>>();
  out[(*count)++] = planes_entry<PlaneCfg<50, float>>();
  out[(*count)++] = planes_entry<PlaneCfg<54, float>>();
  out[(*count)++] = planes_entry<PlaneCfg<60, float>>();
  out[(*count)++] = planes_entry<PlaneCfg<64, float>>();
}
}  // namespace pgj
