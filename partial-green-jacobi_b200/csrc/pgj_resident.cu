// Host side of the cluster-resident PCG (pgj_resident.cuh): the table of built shapes, whether the
// device can co-schedule a grid's clusters, and the launch.
#include "pgj_resident.cuh"
#include <cstdlib>

namespace pgj {

void resident_f64a(ResidentKernel* out, int* count);
void resident_f64b(ResidentKernel* out, int* count);
void resident_f32a(ResidentKernel* out, int* count);
void resident_f32b(ResidentKernel* out, int* count);

namespace {
constexpr int kMaxResident = 64;
struct Table {
  ResidentKernel k[kMaxResident];
  int count = 0;
  Table() {
    resident_f64a(k, &count);
    resident_f64b(k, &count);
    resident_f32a(k, &count);
    resident_f32b(k, &count);
  }
};
const Table& table() {
  static const Table t;
  return t;
}

cudaLaunchConfig_t config(const ResidentKernel& k, int loads, cudaLaunchAttribute* at, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(k.cl * loads));
  cfg.blockDim = dim3(unsigned(k.nt));
  cfg.dynamicSmemBytes = k.smem;
  cfg.stream = s;
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = unsigned(k.cl);
  at->val.clusterDim.y = 1;
  at->val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}
}  // namespace

const ResidentKernel* resident_find(int n, int prec) {
  const Table& t = table();
  for (int i = 0; i < t.count; ++i)
    if (t.k[i].n == n && t.k[i].prec == prec) return &t.k[i];
  return nullptr;
}

size_t resident_halo_bytes(int n, int prec) {
  const ResidentKernel* k = resident_find(n, prec);
  return k ? k->halo : 0;
}

// Sets the kernel's launch limits on the current device and asks whether one cluster can be resident
// there at all (a device partition may have too few SMs in a cluster's reach). Asked for every context: the
// limits go with the device's CUDA context when that is replaced (cudaDeviceReset).
const ResidentKernel* resident_prepare(int n, int prec) {
  const char* e = std::getenv("PGJ_RESIDENT");
  if (e && e[0] == '0') return nullptr;
  const ResidentKernel* k = resident_find(n, prec);
  if (!k) return nullptr;
  cudaError_t err = cudaFuncSetAttribute(k->fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(k->smem));
  if (err == cudaSuccess && k->cl > 8)
    err = cudaFuncSetAttribute(k->fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  int clusters = 0;
  if (err == cudaSuccess) {
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t cfg = config(*k, 1, &at, nullptr);
    err = cudaOccupancyMaxActiveClusters(&clusters, k->fn, &cfg);
  }
  if (err != cudaSuccess) cudaGetLastError();  // not launchable here: the separate kernels serve
  return err == cudaSuccess && clusters >= 1 ? k : nullptr;
}

template <typename T>
__global__ void k_scale_planes(size_t N, const double* __restrict__ s, T* __restrict__ out) {
  scale_planes_row(N, blockIdx.y, s, out);
}

// Self-test: an mbarrier that nothing arrives at.
__global__ void k_cluster_wait_selftest(long long limit, int* flag) {
  __shared__ ClusterBar bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar.tx[0], 1);
    fence_mbar_init();
    bar.dead = 0;
  }
  __syncthreads();
  cluster_wait_on(&bar, &bar.tx[0], 0u, limit);
  __syncthreads();
  if (threadIdx.x == 0) *flag = bar.dead;
}

int launch_cluster_wait_selftest(int limit_us, int* flag, cudaStream_t s) {
  const long long limit = 1000ll * limit_us;
  k_cluster_wait_selftest<<<1, 32, 0, s>>>(limit < kClusterWaitClocks ? limit : kClusterWaitClocks, flag);
  return check_launch();
}

int launch_scale_planes(pgj_ctx* c, int loads, cudaStream_t s) {
  const size_t N = size_t(c->N);
  const dim3 grid(unsigned((N + 255) / 256 < 148 ? (N + 255) / 256 : 148), unsigned((loads + c->lpd - 1) / c->lpd));
  if (c->prec == PGJ_FP32) k_scale_planes<float><<<grid, 256, 0, s>>>(N, c->scale, c->scale32);
  else k_scale_planes<double><<<grid, 256, 0, s>>>(N, c->scale, c->scale_pl);
  return check_launch();
}

int launch_resident(pgj_ctx* c, int loads, cudaStream_t s) {
  const ResidentKernel& k = *c->res;
  const bool f32 = c->prec == PGJ_FP32;
  int st = launch_scale_planes(c, loads, s);
  if (st) return st;
  ResidentArgs A;
  A.lpd = c->lpd; A.cap = c->cap; A.loads = loads;
  A.a = c->a;
  A.f = c->f; A.x = c->x;
  A.q = c->q; A.spec = c->spec; A.q64 = c->r64;
  A.halo = c->halo; A.out = c->scal_out; A.counters = c->cond; A.rel_delta2 = c->rel_delta2; A.kc = c->kc;
  if (f32) {
    A.sp = c->scale32; A.sym = c->symbol32; A.tw = static_cast<double2*>(c->tw) + c->n;
    A.r0 = c->r64; A.r = c->r; A.d = c->d; A.p = c->p;
  } else {
    A.sp = c->scale_pl; A.sym = c->symbol; A.tw = c->tw;
    A.r0 = static_cast<const double*>(c->r); A.r = c->sw; A.d = c->d; A.p = c->p;
  }
  cudaLaunchAttribute at;
  const cudaLaunchConfig_t cfg = config(k, loads, &at, s);
  void* args[] = {&A};
  const cudaError_t e = cudaLaunchKernelExC(&cfg, k.fn, args);
  return e == cudaSuccess ? PGJ_OK : set_cuda_error(e);
}

}  // namespace pgj
