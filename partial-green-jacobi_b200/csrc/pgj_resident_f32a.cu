// Cluster-resident PCG kernels, FP32 recurrences, grids up to 24 (shapes: pgj_resident.cuh).
#include "pgj_resident.cuh"

namespace pgj {
void resident_f32a(ResidentKernel* out, int* count) {
  //                               N    type   CL  TY   NT  PG  CS   p     q     direct
  out[(*count)++] = resident_entry<ResidentCfg<8, float, 4, 8, 64, 3, 10, true, true, true>>();
  out[(*count)++] = resident_entry<ResidentCfg<10, float, 5, 10, 192, 3, 12, true, true, true>>();
  out[(*count)++] = resident_entry<ResidentCfg<12, float, 6, 12, 256, 3, 14, true, true, true>>();
  out[(*count)++] = resident_entry<ResidentCfg<16, float, 8, 16, 256, 3, 18, true, true, true>>();
  out[(*count)++] = resident_entry<ResidentCfg<18, float, 9, 18, 352, 3, 20, true, true, true>>();
  out[(*count)++] = resident_entry<ResidentCfg<20, float, 10, 10, 256, 3, 22, true, true, true>>();
  out[(*count)++] = resident_entry<ResidentCfg<24, float, 12, 12, 288, 3, 26, true, true, true>>();
}
}  // namespace pgj
