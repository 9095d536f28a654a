// Host side of the plane transform kernels (pgj_planes.cuh): the table of built grids and the launches.
//
// Measured, three kernels per iteration (forward / z / inverse), six loads, one B200, us, against the row-packed
// slab kernels and per-line z passes that these replaced (or, where their slab did not fit, the seven
// step-by-step kernels): FP64 n = 48 21 / 21 / 14 against 59 / 35 / 33; n = 64 52 / 28 / 41 against
// 91 / 64 / 50 (the old forward kernel carried the iterate's update, which the inverse one does now);
// n = 80 108 / 75 / 99 against 254 / 162 / 126; n = 96 185 / 113 / 168 against 1049. FP32 n = 48
// 19 / 17 / 10 against 40 / 31 / 27; n = 64 25 / 21 / 19 against 47 / 35 / 27; n = 96 87 / 61 / 83 against
// 178 / 131 / 123; n = 128 235 / 178 / 216 against 1307.
#include "pgj_planes.cuh"
#include <cstring>

namespace pgj {

void planes_f64a(PlaneKernels* out, int* count);
void planes_f64b(PlaneKernels* out, int* count);
void planes_f64c(PlaneKernels* out, int* count);
void planes_f32a(PlaneKernels* out, int* count);
void planes_f32b(PlaneKernels* out, int* count);
void planes_f32c(PlaneKernels* out, int* count);

namespace {
constexpr int kMaxPlanes = 64;
struct Table {
  PlaneKernels k[kMaxPlanes];
  int count = 0;
  Table() {
    planes_f64a(k, &count);
    planes_f64b(k, &count);
    planes_f64c(k, &count);
    planes_f32a(k, &count);
    planes_f32b(k, &count);
    planes_f32c(k, &count);
  }
};
const Table& table() {
  static const Table t;
  return t;
}
}  // namespace

const PlaneKernels* planes_find(int n, int prec) {
  const Table& t = table();
  for (int i = 0; i < t.count; ++i)
    if (t.k[i].n == n && t.k[i].prec == prec) return &t.k[i];
  return nullptr;
}

bool fused_selectable(int n, int prec) {
  const size_t ns = size_t(n / 2 + 1), nsp = ns + (ns & 1);
  return planes_find(n, prec) && 4 * size_t(n) * nsp * (prec == PGJ_FP32 ? 4 : 8) <= 110 * 1024;
}

// Shared memory limits of a grid's kernels on the current device. Set for every context: they go with the device's
// CUDA context when that is replaced (cudaDeviceReset).
int planes_prepare(const PlaneKernels* k) {
  cudaError_t e = cudaFuncSetAttribute(k->fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, int(k->smem));
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k->inv, cudaFuncAttributeMaxDynamicSharedMemorySize, int(k->smem));
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k->z, cudaFuncAttributeMaxDynamicSharedMemorySize, int(k->zsmem));
  return e == cudaSuccess ? PGJ_OK : set_cuda_error(e);
}

static PlaneArgs plane_args(pgj_ctx* c, int loads) {
  const bool f32 = c->prec == PGJ_FP32;
  PlaneArgs A;
  std::memset(&A, 0, sizeof(A));
  A.lpd = c->lpd; A.loads = loads; A.cap = c->cap;
  A.flex = f32 ? c->flex : 0;
  A.p = c->p; A.q = c->q; A.d = c->d;
  A.r = f32 ? c->r : c->sw;  // FP64: c->r holds the certified residual, node-major
  A.r64 = f32 ? c->r64 : static_cast<const double*>(c->r);
  A.sp = f32 ? static_cast<const void*>(c->scale32) : static_cast<const void*>(c->scale_pl);
  A.spec = c->spec; A.shat = c->shat;
  A.zprev = c->sw;  // FP32 only
  A.sym = f32 ? static_cast<const void*>(c->symbol32) : static_cast<const void*>(c->symbol);
  A.tw = f32 ? static_cast<const void*>(static_cast<double2*>(c->tw) + c->n) : c->tw;
  A.scal = c->scal; A.out = c->scal_out; A.partials = c->partials;
  A.rel_delta2 = c->rel_delta2; A.counters = c->cond;
  return A;
}

static int launch(const void* fn, dim3 grid, int threads, size_t smem, PlaneArgs& A, cudaStream_t s) {
  void* args[] = {&A};
  const cudaError_t e = cudaLaunchKernel(fn, grid, dim3(unsigned(threads)), args, smem, s);
  return e == cudaSuccess ? PGJ_OK : set_cuda_error(e);
}

static dim3 plane_grid(const pgj_ctx* c, int loads) { return dim3(3, unsigned(c->n / 2), unsigned(loads)); }
static dim3 line_grid(const PlaneKernels& k, int loads) { return dim3(unsigned((k.m + k.cs - 1) / k.cs), unsigned(loads)); }

int launch_planes_fwd(pgj_ctx* c, int loads, int mode, cudaStream_t s, cudaGraphConditionalHandle hif) {
  PlaneArgs A = plane_args(c, loads);
  A.h = hif;
  A.set_cond = hif ? 1 : 0;
  A.mode = mode;
  return launch(c->planes->fwd, plane_grid(c, loads), c->planes->nt, c->planes->smem, A, s);
}

int launch_planes_z(pgj_ctx* c, int loads, bool init, cudaStream_t s) {
  PlaneArgs A = plane_args(c, loads);
  A.init = init ? 1 : 0;
  return launch(c->planes->z, line_grid(*c->planes, loads), c->planes->zt, c->planes->zsmem, A, s);
}

int launch_planes_inv(pgj_ctx* c, int loads, bool init, cudaStream_t s, cudaGraphConditionalHandle h, bool set_cond) {
  PlaneArgs A = plane_args(c, loads);
  A.init = init ? 1 : 0;
  A.set_cond = set_cond ? 1 : 0;
  A.h = h;
  return launch(c->planes->inv, plane_grid(c, loads), c->planes->nt, c->planes->smem, A, s);
}

// What the apply needs beforehand, in one launch: rows y < designs of the grid copy the designs' scale fields by
// component, the others form the means of the loads' vectors (n = 64, six loads: 139.4 us without the means, 141.1
// with them).
static __global__ void __launch_bounds__(256) k_apply_prepare(size_t N, int designs, const double* __restrict__ scale,
                                                              double* __restrict__ sp, const double* __restrict__ r,
                                                              LoadScalars* scal, double* partials) {
  if (int(blockIdx.y) < designs) {
    scale_planes_row(N, blockIdx.y, scale, sp);
    return;
  }
  const int load = int(blockIdx.y) - designs;
  grid_mean3(N, r + size_t(load) * 3 * N, scal[load].mean_r, scal[load], partials + size_t(load) * kPartialQ * kMaxPartials);
}

int launch_planes_apply(pgj_ctx* c, int loads, const double* r, double* z, cudaStream_t s) {
  const int designs = (loads + c->lpd - 1) / c->lpd;
  k_apply_prepare<<<dim3(148, unsigned(designs + loads)), 256, 0, s>>>(size_t(c->N), designs, c->scale, c->scale_pl, r,
                                                                       c->scal, c->partials);
  int st = check_launch();
  if (!st) st = launch_planes_shat(c, loads, s);
  PlaneArgs A = plane_args(c, loads);
  A.mode = kPlanesApply;
  A.init = 1;
  A.r64 = r;
  A.z64 = z;
  const PlaneKernels& k = *c->planes;
  if (!st) st = launch(k.fwd, plane_grid(c, loads), k.nt, k.smem, A, s);
  if (!st) st = launch(k.z, line_grid(k, loads), k.zt, k.zsmem, A, s);
  return st ? st : launch(k.inv, plane_grid(c, loads), k.nt, k.smem, A, s);
}

// DFT(s) of the designs of `loads` loads, from the scale copy by component.
int launch_planes_shat(pgj_ctx* c, int loads, cudaStream_t s) {
  const int designs = (loads + c->lpd - 1) / c->lpd;
  PlaneArgs A = plane_args(c, loads);
  A.mode = kPlanesScale;
  A.spec = c->shat;
  int st = launch(c->planes->fwd, plane_grid(c, designs), c->planes->nt, c->planes->smem, A, s);
  if (st) return st;
  A.forward_only = 1;
  return launch(c->planes->z, line_grid(*c->planes, designs), c->planes->zt, c->planes->zsmem, A, s);
}

}  // namespace pgj
