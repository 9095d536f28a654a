// Cluster-resident PCG kernels, FP64, grids from 30 (shapes: pgj_resident.cuh).
#include "pgj_resident.cuh"

namespace pgj {
void resident_f64b(ResidentKernel* out, int* count) {
  //                               N    type    CL  TY   NT  PG  CS   p     q     direct
  out[(*count)++] = resident_entry<ResidentCfg<30, double, 15, 10, 320, 3, 32, true, true, true>>();
  out[(*count)++] = resident_entry<ResidentCfg<32, double, 16, 8, 384, 3, 34, true, true, true>>();
  out[(*count)++] = resident_entry<ResidentCfg<36, double, 12, 12, 512, 5, 57, false, true, false>>();
  out[(*count)++] = resident_entry<ResidentCfg<48, double, 16, 8, 384, 5, 75, false, false, false>>();
}
}  // namespace pgj
