// Plane transform kernels, FP64, grids up to 36 (pgj_planes.cuh).
#include "pgj_planes.cuh"

namespace pgj {
void planes_f64a(PlaneKernels* out, int* count) {
  out[(*count)++] = planes_entry<PlaneCfg<4, double>>();
  out[(*count)++] = planes_entry<PlaneCfg<6, double>>();
  out[(*count)++] = planes_entry<PlaneCfg<8, double>>();
  out[(*count)++] = planes_entry<PlaneCfg<10, double>>();
  out[(*count)++] = planes_entry<PlaneCfg<12, double>>();
  out[(*count)++] = planes_entry<PlaneCfg<16, double>>();
  out[(*count)++] = planes_entry<PlaneCfg<18, double>>();
  out[(*count)++] = planes_entry<PlaneCfg<20, double>>();
  out[(*count)++] = planes_entry<PlaneCfg<24, double>>();
  out[(*count)++] = planes_entry<PlaneCfg<30, double>>();
  out[(*count)++] = planes_entry<PlaneCfg<32, double>>();
  out[(*count)++] = planes_entry<PlaneCfg<36, double>>();
}
}  // namespace pgj
