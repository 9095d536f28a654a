// Cluster-resident PCG kernels, FP64, grids 30 and 32 (shapes: pgj_resident.cuh).
#include "pgj_resident.cuh"

namespace pgj {
void resident_f64b(ResidentKernel* out, int* count) {
  //                               N    type    CL  TY   NT  PG  CS   p     q     direct
  out[(*count)++] = resident_entry<ResidentCfg<30, double, 15, 10, 320, 3, 32, true, true, true>>();
  out[(*count)++] = resident_entry<ResidentCfg<32, double, 16, 8, 384, 3, 34, true, true, true>>();
}
}  // namespace pgj
