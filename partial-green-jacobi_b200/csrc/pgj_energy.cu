// Element strain energies and the homogenized tensor.
//
// For v_l = u_l + A_l on an element (A_l the affine field of the macro strain), the element
// energy v_i^T Ke v_j equals sum_m Q_i[m] . P_j[m] in the modal basis (the Hadamard transform is
// orthogonal up to the same factor on both sides), with P_j the modal element action for a = 1.
// One pass over the elements therefore gives every pair at once:
//   e_l(el)  = v_l^T Ke v_l / h^3                      (energy.cu:7-24 in exp/asg_scenarios_20261105)
//   C_ij     = mean_el( a v_i^T Ke v_j ) / h^3          (polarisation in reproduction.py:166-176)
#include "pgj_internal.h"

namespace pgj {

struct EnergyArgs {
  int n, loads;
  int zc;                // element planes per block
  const double* u;       // (loads, 3N)
  const double* macros;  // (loads, 6) device
  const double* a;       // (N)
  double* e;             // (loads, N): energies
  double* C;             // 36: tensor
  LoadScalars* scal;     // ticket owner (record 0)
  double* partials;      // 21 * kMaxPartials
  OpConst kc;            // a = 1 constants of C0
};

constexpr int kEnergyLanes = 32;     // elements of a plane per block of the tensor kernel, six warps: one per load
constexpr int kEnergyThreads = 128;  // elements of a plane per block of the energy kernel

// Both kernels march planes of elements along z: a thread owns one column of elements of one load and keeps the
// transform of its lower face, so a step reads one face (4 nodes). They are bound by the latency of these loads
// and by FP64 arithmetic. Holding whole elements in shared memory for all loads, one thread per element, left
// 192 threads on an SM and read every node 8 times. Six loads, us, that form / this one: tensor n = 32 56 / 14,
// 54 127 / 37, 96 622 / 161; energies 54 46 / 17, 96 313 / 74.

// x/y transform of the four nodes of a face of the column, per component
struct EnergyColumn {
  const double* u;            // the load's vector
  unsigned o00, o10, o01, o11, plane;
  __device__ EnergyColumn(const double* ul, int n, int x, int y) : u(ul), plane(3u * n * n) {
    const unsigned x1 = x + 1 == n ? 0 : x + 1, y1 = y + 1 == n ? 0 : y + 1;
    o00 = 3u * (unsigned(y) * n + x); o10 = 3u * (unsigned(y) * n + x1);
    o01 = 3u * (y1 * n + x); o11 = 3u * (y1 * n + x1);
  }
  __device__ __forceinline__ void face(unsigned z, double (&F)[4][3]) const {
    const double* p = u + z * plane;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double v00 = __ldg(p + o00 + c), v10 = __ldg(p + o10 + c);
      const double v01 = __ldg(p + o01 + c), v11 = __ldg(p + o11 + c);
      const double s0 = v10 + v00, d0 = v10 - v00, s1 = v11 + v01, d1 = v11 - v01;
      F[0][c] = s1 + s0; F[1][c] = d1 + d0; F[2][c] = s1 - s0; F[3][c] = d1 - d0;
    }
  }
};

// Modes of u + the affine field of the macro strain m on the element between the faces F0 (below) and F1, which
// becomes the lower face of the next. The affine field is in the first-order modes only: 4 h E.
__device__ __forceinline__ void energy_modes(const EnergyColumn& col, unsigned z, const double (&E)[6], double (&F0)[4][3],
                                             double (&Q)[8][3]) {
  double F1[4][3];
  col.face(z, F1);
#pragma unroll
  for (int f = 0; f < 4; ++f)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      Q[f][c] = F1[f][c] + F0[f][c];
      Q[f + 4][c] = F1[f][c] - F0[f][c];
      F0[f][c] = F1[f][c];
    }
  Q[1][0] += E[0]; Q[1][1] += E[5]; Q[1][2] += E[4];
  Q[2][0] += E[5]; Q[2][1] += E[1]; Q[2][2] += E[3];
  Q[4][0] += E[4]; Q[4][1] += E[3]; Q[4][2] += E[2];
}

// 4 h times the symmetric tensor (xx, yy, zz, yz, xz, xy) of an engineering Voigt strain
__device__ __forceinline__ void energy_strain(const double* m, int n, double (&E)[6]) {
  const double h4 = 4.0 / n;
#pragma unroll
  for (int k = 0; k < 6; ++k) E[k] = (k < 3 ? m[k] : m[k] / 2) * h4;
}

__device__ __forceinline__ double energy_dot(const double (&Q)[8][3], const double (&P)[8][3]) {
  double s = 0.0;
#pragma unroll
  for (int m = 1; m < 8; ++m)
#pragma unroll
    for (int c = 0; c < 3; ++c) s += Q[m][c] * P[m][c];
  return s;
}

// Energies of one load per blockIdx.y, z chunk per blockIdx.z.
__global__ void __launch_bounds__(kEnergyThreads) k_energies(const EnergyArgs A) {
  const int n = A.n, load = blockIdx.y;
  const unsigned nn = unsigned(n) * n, i = blockIdx.x * kEnergyThreads + threadIdx.x;
  if (i >= nn) return;
  const size_t N = size_t(nn) * n;
  const int z0 = blockIdx.z * A.zc, z1 = min(z0 + A.zc, n);
  const EnergyColumn col(A.u + size_t(load) * 3 * N, n, int(i % n), int(i / n));
  double E[6], F0[4][3];
  energy_strain(A.macros + 6 * load, n, E);
  const double invv = double(n) * n * n;
  col.face(z0, F0);
  double* e = A.e + size_t(load) * N + i;
#pragma unroll 1
  for (int z = z0; z < z1; ++z) {
    double Q[8][3], P[8][3];
    energy_modes(col, z + 1 == n ? 0 : z + 1, E, F0, Q);
    element_modal<double>(Q, 1.0, A.kc, P);
    e[size_t(z) * nn] = energy_dot(Q, P) * invv;
  }
}

// Tensor of six loads: warp j owns load j. It publishes its modes, double-buffered
// over one barrier a step, and takes the pairs (j, j + k mod 6), k = 0, 1, 2, the first three warps also k = 3: each
// of the 21 pairs once, so that the warps' work differs by one pair. Two blocks per SM: 158 registers; with three
// the compiler has 96 and spills.
__global__ void __launch_bounds__(6 * kEnergyLanes, 2) k_tensor(const EnergyArgs A) {
  const int n = A.n, lane = threadIdx.x, j = threadIdx.y;
  const unsigned nn = unsigned(n) * n, i0 = blockIdx.x * kEnergyLanes + lane, i = i0 < nn ? i0 : 0;
  const size_t N = size_t(nn) * n;
  const int z0 = blockIdx.y * A.zc, z1 = min(z0 + A.zc, n);
  extern __shared__ double Qsm[];  // [parity][load][mode, component][lane]
  constexpr int kLoad = 21 * kEnergyLanes;
  const EnergyColumn col(A.u + size_t(j) * 3 * N, n, int(i % n), int(i / n));
  double E[6], F0[4][3];
  energy_strain(A.macros + 6 * j, n, E);
  const double invv = double(n) * n * n;
  col.face(z0, F0);
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 1
  for (int z = z0; z < z1; ++z) {
    const double ae = i0 < nn ? __ldg(A.a + size_t(z) * nn + i) : 0.0;
    double* buf = Qsm + ((z - z0) & 1) * 6 * kLoad + lane;
    double Q[8][3], P[8][3];
    energy_modes(col, z + 1 == n ? 0 : z + 1, E, F0, Q);
#pragma unroll
    for (int m = 1; m < 8; ++m)
#pragma unroll
      for (int c = 0; c < 3; ++c) buf[j * kLoad + ((m - 1) * 3 + c) * kEnergyLanes] = Q[m][c];
    element_modal<double>(Q, 1.0, A.kc, P);
    acc[0] += ae * energy_dot(Q, P);
    __syncthreads();  // modes published; the other parity's have been read
#pragma unroll
    for (int k = 1; k < 4; ++k) {
      if (k == 3 && j >= 3) continue;
      const double* q = buf + (j + k < 6 ? j + k : j + k - 6) * kLoad;
      double s = 0.0;
#pragma unroll
      for (int m = 1; m < 8; ++m)
#pragma unroll
        for (int c = 0; c < 3; ++c) s += q[((m - 1) * 3 + c) * kEnergyLanes] * P[m][c];
      acc[k] += ae * s;
    }
  }
  const int blk = blockIdx.x + gridDim.x * blockIdx.y, nblk = gridDim.x * gridDim.y;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (k == 3 && j >= 3) continue;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_down_sync(0xffffffffu, acc[k], o);
    if (lane == 0) A.partials[size_t(6 * k + j) * kMaxPartials + blk] = acc[k];
  }
  if (!last_block(&A.scal[0].ticket[kTicketAux2], nblk)) return;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (k == 3 && j >= 3) continue;
    const double* part = A.partials + size_t(6 * k + j) * kMaxPartials;
    double s = 0.0;
    for (int b = lane; b < nblk; b += 32) s += __ldcg(part + b);
    s = warp_reduce(s, lane, 32);
    if (lane == 0) {
      const int o = j + k < 6 ? j + k : j + k - 6;
      const double v = s * invv / double(N);
      A.C[o * 6 + j] = v;
      A.C[j * 6 + o] = v;
    }
  }
}

// z chunks: the most even filling of the chip's `slots` blocks, counting the face that a chunk reads beyond its own;
// at most `most` blocks.
static int energy_chunk(int n, long columns, long slots, long most) {
  double top = -1.0;
  int best = n;
  for (int nch = 1; nch <= (n + 3) / 4; ++nch) {
    const int zc = (n + nch - 1) / nch, chunks = (n + zc - 1) / zc;
    const long blocks = columns * chunks, waves = (blocks + slots - 1) / slots;
    if (blocks > most) break;
    const double eff = double(n) / (double(chunks) * (zc + 1)) * double(blocks) / double(waves * slots);
    if (eff > top + 1e-9) { top = eff; best = zc; }
  }
  return best;
}

static int launch_tensor(EnergyArgs& A, cudaStream_t s) {
  const int n = A.n;
  const unsigned columns = unsigned((n * n + kEnergyLanes - 1) / kEnergyLanes);
  A.zc = energy_chunk(n, columns, 2 * 148, kMaxPartials);
  const size_t smem = size_t(2) * 6 * 21 * kEnergyLanes * sizeof(double);
  const cudaError_t e = cudaFuncSetAttribute(k_tensor, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  if (e != cudaSuccess) return set_cuda_error(e);
  k_tensor<<<dim3(columns, unsigned((n + A.zc - 1) / A.zc)), dim3(kEnergyLanes, 6), smem, s>>>(A);
  return check_launch();
}

static EnergyArgs energy_args(pgj_ctx* c, int loads, const double* u, const double* macros_dev) {
  EnergyArgs A;
  A.n = c->n; A.loads = loads; A.u = u; A.macros = macros_dev; A.a = c->a;
  A.e = nullptr; A.C = nullptr; A.scal = c->scal; A.partials = c->partials;
  A.kc = make_opconst(c->n, c->lam, c->mu);
  return A;
}

int launch_energies(pgj_ctx* c, int loads, const double* u, const double* macros_dev, double* e, cudaStream_t s) {
  if (loads < 1 || loads > kMaxLoads) return PGJ_ERR_ARGUMENT;
  EnergyArgs A = energy_args(c, loads, u, macros_dev);
  A.e = e;
  const unsigned columns = unsigned((c->n * c->n + kEnergyThreads - 1) / kEnergyThreads);
  A.zc = energy_chunk(c->n, long(columns) * loads, 4 * 148, 1L << 40);
  k_energies<<<dim3(columns, loads, unsigned((c->n + A.zc - 1) / A.zc)), kEnergyThreads, 0, s>>>(A);
  return check_launch();
}

int launch_effective_tensor(pgj_ctx* c, const double* a, const double* u, double* C, cudaStream_t s) {
  EnergyArgs A = energy_args(c, 6, u, c->aux + kAuxVoigt);  // unit Voigt macros (6 x 6)
  A.a = a;
  A.C = C;
  return launch_tensor(A, s);
}

}  // namespace pgj

// ------------------------------------------------------------------------------------------------
// Homogenized tensor without any device allocation by the caller or the library.
//
// Some callers cannot allocate device memory: a host application that owns the whole device
// memory pool and forbids third-party cudaMalloc (for instance a finite-element code that calls
// this library as a post-processing plugin inside its own memory budget). They still hold the
// density field and the six solutions, and want C_H from them. This entry point runs the same C_H
// kernel as pgj_effective_tensor, with its scratch (block partial sums and the last-block ticket)
// in a fixed file-scope device array instead of a context workspace; the six unit Voigt strains
// are a statically initialised device table, so nothing has to be copied before the first call.
//
// Limits and sharing: the array is kNoAllocScratchBytes (about 0.69 MB) on every GPU that loads
// the library, held until the process exits; it fits the kernel's partial sums for any grid the
// entry point accepts (2 <= n <= 256). Every call on a device uses the same array and the array
// keeps the last call's contents; the ticket is cleared at the start of each call. Two calls whose
// work overlaps on the GPU (for example on two streams without ordering) race on the array and
// give wrong results: order them on one stream or synchronise between them.
#include <mutex>

namespace {
constexpr size_t kNoAllocPartialDoubles = size_t(21) * pgj::kMaxPartials;
constexpr size_t kNoAllocScalarBytes = 256;
constexpr size_t kNoAllocScratchBytes = kNoAllocPartialDoubles * sizeof(double) + kNoAllocScalarBytes;
static_assert(sizeof(pgj::LoadScalars) <= kNoAllocScalarBytes, "scalar record must fit its slot");

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];
// (6, 6) unit engineering Voigt strains, one row per load
static __device__ const double g_noalloc_voigt[36] = {1, 0, 0, 0, 0, 0, 0, 1, 0, 0, 0, 0, 0, 0, 1, 0, 0, 0,
                                                      0, 0, 0, 1, 0, 0, 0, 0, 0, 0, 1, 0, 0, 0, 0, 0, 0, 1};

// Device addresses of the two symbols, looked up once per device with that device current and
// kept together with the id of the context they belong to: a replaced context (cudaDeviceReset,
// a new primary context) has another id, and the lookup is redone. The host-side names of the
// symbols are stand-ins, never passed to a kernel. A mutex orders first calls from several threads.
constexpr int kNoAllocMaxDevices = 64;
struct NoAllocSlot {
  unsigned long long ctx_id = 0;
  unsigned char* scratch = nullptr;
  const double* voigt = nullptr;
};
NoAllocSlot g_noalloc_slot[kNoAllocMaxDevices];
std::mutex g_noalloc_mutex;

// Current context id through the driver entry points the runtime exposes (no libcuda link).
// Returns 0 when the thread has no current context yet.
unsigned long long current_context_id() {
  using GetCurrent = int (*)(void**);
  using GetId = int (*)(void*, unsigned long long*);
  static GetCurrent get_current = nullptr;
  static GetId get_id = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_current = reinterpret_cast<GetCurrent>(f);
    if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_id = reinterpret_cast<GetId>(f);
  });
  void* ctx = nullptr;
  unsigned long long id = 0;
  if (!get_current || !get_id || get_current(&ctx) != 0 || !ctx || get_id(ctx, &id) != 0) return 0;
  return id;
}

int noalloc_setup(int device, unsigned char** scratch, const double** voigt) {
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  NoAllocSlot& slot = g_noalloc_slot[device];
  unsigned long long id = current_context_id();
  if (id != 0 && slot.ctx_id == id && slot.scratch) {
    *scratch = slot.scratch;
    *voigt = slot.voigt;
    return PGJ_OK;
  }
  void* p = nullptr;
  void* v = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
  if (e == cudaSuccess) e = cudaGetSymbolAddress(&v, g_noalloc_voigt);
  if (e != cudaSuccess) return pgj::set_cuda_error(e);
  if (id == 0) id = current_context_id();  // the lookup made the device's context current
  slot.ctx_id = id;
  slot.scratch = static_cast<unsigned char*>(p);
  slot.voigt = static_cast<const double*>(v);
  *scratch = slot.scratch;
  *voigt = slot.voigt;
  return PGJ_OK;
}
}  // namespace

extern "C" int pgj_effective_tensor_noalloc(int n, double lam, double mu, const double* a, const double* u,
                                            double* C, void* stream) {
  if (n < 2 || n > 256) return PGJ_ERR_ARGUMENT;  // beyond the grids this scratch is sized for
  if (!a || !u || !C || !(mu > 0) || !(lam + 2 * mu / 3 > 0)) return PGJ_ERR_ARGUMENT;
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return pgj::set_cuda_error(e);
  if (device < 0 || device >= kNoAllocMaxDevices) return PGJ_ERR_UNSUPPORTED;
  unsigned char* base = nullptr;
  const double* voigt = nullptr;
  int st = noalloc_setup(device, &base, &voigt);
  if (st) return st;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  double* partials = reinterpret_cast<double*>(base);
  pgj::LoadScalars* scal = reinterpret_cast<pgj::LoadScalars*>(partials + kNoAllocPartialDoubles);
  // the last-block ticket must start at zero
  e = cudaMemsetAsync(scal, 0, sizeof(pgj::LoadScalars), s);
  if (e != cudaSuccess) return pgj::set_cuda_error(e);
  pgj::EnergyArgs A;
  A.n = n; A.loads = 6; A.u = u; A.macros = voigt; A.a = a;
  A.e = nullptr; A.C = C; A.scal = scal; A.partials = partials;
  A.kc = pgj::make_opconst(n, lam, mu);
  return pgj::launch_tensor(A, s);
}
