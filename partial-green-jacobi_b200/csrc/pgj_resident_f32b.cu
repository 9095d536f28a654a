// Cluster-resident PCG kernels, FP32 recurrences, grids 30 to 36 (shapes: pgj_resident.cuh).
#include "pgj_resident.cuh"

namespace pgj {
void resident_f32b(ResidentKernel* out, int* count) {
  //                               N    type   CL  TY   NT  PG  CS   p     q     direct
  out[(*count)++] = resident_entry<ResidentCfg<30, float, 15, 10, 320, 3, 32, true, true, true>>();
  out[(*count)++] = resident_entry<ResidentCfg<32, float, 16, 8, 384, 3, 34, true, true, true>>();
  out[(*count)++] = resident_entry<ResidentCfg<36, float, 12, 6, 384, 5, 57, true, true, false>>();
}
}  // namespace pgj
