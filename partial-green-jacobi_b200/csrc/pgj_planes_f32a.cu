// Plane transform kernels, FP32, grids up to 36 (pgj_planes.cuh).
#include "pgj_planes.cuh"

namespace pgj {
void planes_f32a(PlaneKernels* out, int* count) {
  out[(*count)++] = planes_entry<PlaneCfg<4, float>>();
  out[(*count)++] = planes_entry<PlaneCfg<6, float>>();
  out[(*count)++] = planes_entry<PlaneCfg<8, float>>();
  out[(*count)++] = planes_entry<PlaneCfg<10, float>>();
  out[(*count)++] = planes_entry<PlaneCfg<12, float>>();
  out[(*count)++] = planes_entry<PlaneCfg<16, float>>();
  out[(*count)++] = planes_entry<PlaneCfg<18, float>>();
  out[(*count)++] = planes_entry<PlaneCfg<20, float>>();
  out[(*count)++] = planes_entry<PlaneCfg<24, float>>();
  out[(*count)++] = planes_entry<PlaneCfg<30, float>>();
  out[(*count)++] = planes_entry<PlaneCfg<32, float>>();
  out[(*count)++] = planes_entry<PlaneCfg<36, float>>();
}
}  // namespace pgj
