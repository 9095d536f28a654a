// Plane transform kernels, FP64, grids from 40 to 64 (pgj_planes.cuh).
#include "pgj_planes.cuh"

namespace pgj {
void planes_f64b(PlaneKernels* out, int* count) {
  out[(*count)++] = planes_entry<PlaneCfg<40, double>>();
  out[(*count)++] = planes_entry<PlaneCfg<48, double>>();
  out[(*count)++] = planes_entry<PlaneCfg<50, double>>();
  out[(*count)++] = planes_entry<PlaneCfg<54, double>>();
  out[(*count)++] = planes_entry<PlaneCfg<60, double>>();
  out[(*count)++] = planes_entry<PlaneCfg<64, double>>();
}
}  // namespace pgj
