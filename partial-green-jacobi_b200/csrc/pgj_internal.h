// Internal host-side interfaces shared by the libpgj translation units.
#pragma once
#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>
#include "pgj_common.cuh"

namespace pgj {

struct FFTPlan {
  int n;
  int nst;
  int radix[kMaxStages];
  FastDiv ns_div[kMaxStages];  // stride Ns of each stage (product of the earlier radices)
  FastDiv nb_div[kMaxStages];  // butterflies per line of each stage (n / radix)
};
bool make_fft_plan(int n, FFTPlan* plan);

// Launch geometry of the operator for a grid edge n (rows_geom).
struct StencilGeom {
  int ty;      // output node rows per block (block is n / 2 x (ty + 1) threads)
  int ntiles;  // tiles along y
  int zc;      // output node planes per block
  int nchunks; // chunks along z
  int occ;     // blocks per SM
};
// `wide`: FP64 arithmetic
StencilGeom rows_geom(int n, int lpd, bool wide);

// Geometry of the FFT passes.
struct FFTGeom {
  int rb;        // rows (z,y) per x-pass block
  int kcy;       // kx columns per y-pass block
  int nky;       // y-pass chunks
  int kcz;       // kx columns per z-pass block
  int nkz;       // z-pass chunks
  int thr_x, thr_y, thr_z;  // threads per block of the x, y and z passes
  int by_x, by_y, by_z;     // threads along y (butterflies of a line) per pass; x (and z) index lines
  FastDiv div_3n, div_ns, div_n, div_kcz;
};
FFTGeom fft_geom(int n, int elem_bytes, const FFTPlan& plan, int rb_req = 0, int nky_req = 0, int nkz_req = 0);

enum StencilMode { kPlain = 0, kPCG = 1, kResidual = 2 };

struct StencilArgs {
  int n, ty, zc;
  int lpd;                     // loads per design: load l reads the density of design l / lpd
  const double* a;             // (designs, N)
  const void* in;
  void* out;
  const double* f;             // residual mode: right-hand side
  const int32_t* active_ext;   // plain mode: optional external mask
  const LoadScalars* rel_flags; // residual mode: when set, only loads with rel_flags[l].reliable
  LoadScalars* scal;           // pcg / residual modes
  double* partials;            // [load][4][nblk]
  OpConst kc;
};

// Partial-sum slots per load per kernel (blocks per load upper bound).
constexpr int kMaxPartials = 4096;
constexpr int kPartialQ = 5;
// aux block: [0,24) stiffness diagonal per local node, [32,68) unit Voigt macros,
// [128, 128 + kMaxPartials) scalar-reduction partials of the scale build.
constexpr int kAuxVoigt = 32;
constexpr int kAuxPartials = 128;
constexpr int kAuxDoubles = kAuxPartials + kMaxPartials;

// Component means of one load's node-major vector by the blocks of a grid row (256 threads each), to dst[3].
__device__ __forceinline__ void grid_mean3(size_t N, const double* __restrict__ u, double* dst, LoadScalars& S, double* part) {
  double acc[3] = {0.0, 0.0, 0.0};
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < N; i += size_t(gridDim.x) * blockDim.x) {
    acc[0] += u[3 * i]; acc[1] += u[3 * i + 1]; acc[2] += u[3 * i + 2];
  }
  __shared__ double red[96];
  block_sum<3>(acc, red);
  if (threadIdx.x == 0)
    for (int k = 0; k < 3; ++k) part[k * kMaxPartials + blockIdx.x] = acc[k];
  if (!last_block(&S.ticket[kTicketAux], gridDim.x)) return;
  if (threadIdx.x < 32) {
    double v[3];
    for (int k = 0; k < 3; ++k) v[k] = warp_sum_partials(part + k * kMaxPartials, gridDim.x);
    if (threadIdx.x == 0)
      for (int k = 0; k < 3; ++k) dst[k] = v[k] / double(N);
  }
}

// One design's scale field by component, by the blocks of a grid row: out[c][node] = T(s[3 node + c]).
template <typename T>
__device__ __forceinline__ void scale_planes_row(size_t N, int design, const double* __restrict__ s, T* __restrict__ out) {
  s += size_t(design) * 3 * N;
  out += size_t(design) * 3 * N;
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < N; i += size_t(gridDim.x) * blockDim.x) {
    const double a = s[3 * i], b = s[3 * i + 1], c = s[3 * i + 2];
    out[i] = T(a);
    out[N + i] = T(b);
    out[2 * N + i] = T(c);
  }
}

struct Layout {
  size_t a, scale, scale32, symbol, symbol32, tw, solutions, f, x, r, p, q, sw, spec, shat, partials, scal, macros,
      cond, r64, d, aux, scale_pl, halo, total;
};

struct Graphs;
struct ResidentKernel;
struct PlaneKernels;

}  // namespace pgj

struct pgj_ctx {
  int n, L, prec;
  int D, lpd;          // designs and loads per design (L = D * lpd); a plain context has D = 1
  double lam, mu;
  long long N;
  int ns;
  long long Nh;
  pgj::OpConst kc;
  pgj::FFTPlan plan;
  pgj::StencilGeom geo64, geo32;  // the operator's launches in FP64 and FP32 arithmetic
  pgj::FFTGeom fg;
  pgj::Layout lay;
  char* base;
  size_t bytes;
  // workspace views (per-design fields are D consecutive blocks)
  double* a;           // (D, N)
  double* scale;       // (D, 3N)
  float* scale32;      // FP32 contexts: (D, 3, N) component-planar FP32 copy of scale (first direction)
  double* symbol;
  float* symbol32;
  void* tw;            // n complex twiddles: double2[n] then float2[n]
  double* solutions;   // (L, 3N) fp64 warm starts
  double* f;           // (L, 3N) fp64 right-hand sides
  double* x;           // (L, 3N) fp64 iterate (plain) / refined solution (mixed)
  void* r;             // (L, 3N) T
  void* p;             // (L, 3N) T
  void* q;             // (L, 3N) T
  void* sw;            // (L, 3N) T  s . w (unprojected preconditioned residual); plane kernels in FP64: the residual
  void* spec;          // (L, 3, n, n, nsp) complex T (plane kernels: rows of ns)
  void* shat;          // (D, 3, n, n, nsp) complex T: DFT of each component of the scale field
  double* scale_pl;    // FP64 contexts: (D, 3, N) copy of scale by component
  char* halo;          // per load, the planes its cluster's blocks hand to each other
  const pgj::ResidentKernel* res;  // cluster-resident PCG of this grid and precision, or null
  const pgj::PlaneKernels* planes; // plane transform kernels of this grid and precision, or null
  int four;            // PCG iteration as operator + plane transform kernels (or the resident kernel)
  int fused;           // pgj_fused_iteration: the four-kernel set is selected, on a grid where it may be
  double* partials;    // (L, kPartialQ * kMaxPartials)
  pgj::LoadScalars* scal;  // L records used by the kernels being launched (outer or inner)
  pgj::LoadScalars* scal_out;  // certification / FP64 recurrence records
  pgj::LoadScalars* scal_in;   // mixed refinement: inner FP32 recurrence records
  void* d;             // (L, 3N) T correction of the current attempt
  double* macros;      // (L, 6) device copy
  int* cond;           // device flags (any active)
  double* r64;         // mixed: fp64 residual (L, 3N)
  double* aux;         // (64 + kMaxPartials) doubles: small staged tables and scalar reductions
  double alpha;
  double inner_rtol;
  double rel_delta2;   // mixed reliable updates: replace r when ||r||^2 < rel_delta2 * anchor (0 = off)
  int mixed_mode;      // 0 reliable-update CG, 1 restarted refinement sweeps
  int op64;            // FP32 contexts: the recurrence operator computes in FP64 (FP32 vectors)
  int cap;             // per-load PCG iteration cap (4000, the reference's, unless set)
  int flex;            // FP32 recurrences on the plane kernels: flexible (Polak-Ribiere) beta
  int tile_source;     // FFT tiles: 0 tuned by timing at creation, 1 tile table, 2 environment override
  int fft_req[3];      // requested FFT tiles (rows per x block, y chunks, z chunks)
  int last_refinements;
  int pending_loads;       // loads of the solve enqueued by pgj_solve_async
  int diag_staged;         // stiffness-diagonal constants copied to aux
  int staged_loads;        // macros already on the device
  double staged_macros[6 * pgj::kMaxTotalLoads];
  double alphas[pgj::kMaxDesigns];  // alpha of each design's scale field
  long long last_launches;
  pgj::Graphs* graphs;
};

namespace pgj {
// operator (pgj_rows.cu)
int launch_stencil(pgj_ctx* c, int mode, int loads, int prec, const void* in, void* out, const double* f,
                   const int32_t* active_ext, cudaStream_t s, const LoadScalars* rel_flags = nullptr);
// the recurrence operator q = K p (and alpha = r.z / p.q) of one PCG iteration
inline int launch_recurrence_operator(pgj_ctx* c, int loads, int prec, cudaStream_t s) {
  return launch_stencil(c, kPCG, loads, prec, c->p, c->q, nullptr, nullptr, s);
}
// offline-tuned tile shapes per (n, precision); right-hand side, scale, norms (pgj_operator.cu)
struct TileEntry { int n, prec, rb, nky, nkz; };
bool tile_table(int n, int prec, TileEntry* out);
int launch_rhs(pgj_ctx* c, int loads, const double* macros_dev, double* f, cudaStream_t s);
int launch_scale(pgj_ctx* c, double alpha, cudaStream_t s);
int launch_project_u(pgj_ctx* c, int loads, double* u, cudaStream_t s);
// per-load component means of a DOF vector into scal.mean_u (which=0) or scal.mean_r (which=1)
int launch_mean3(pgj_ctx* c, int loads, const double* v, int which, cudaStream_t s);
int launch_norms(pgj_ctx* c, int loads, const double* f, double rtol, cudaStream_t s);
// fft / green (pgj_fft.cu)
int init_fft_tables(pgj_ctx* c, cudaStream_t s);
int build_symbol(int n, double lam, double mu, double* sym, float* sym32, cudaStream_t s);
int launch_green(pgj_ctx* c, int loads, int prec, const void* r, bool init, cudaStream_t s);
// one Green pass: 0 fft_x, 1 fft_y, 2 fft_z+symbol, 3 ifft_y, 4 ifft_x
int launch_green_pass(pgj_ctx* c, int loads, int prec, const void* r, bool init, int pass, cudaStream_t s);
int launch_green_standalone(pgj_ctx* c, int loads, const double* r, double* z, cudaStream_t s);
// plane transform kernels (pgj_planes.cu)
enum PlanesMode { kPlanesUpdate = 0, kPlanesInit = 1, kPlanesSync = 2, kPlanesScale = 3, kPlanesApply = 4 };
const PlaneKernels* planes_find(int n, int prec);
int planes_prepare(const PlaneKernels* k);
// grids on which pgj_set_fused_iteration selects between the two kernel sets: two planes of transform
// buffers per SM (up to n = 80 in FP64, 108 in FP32). Larger grids whose plane pair fits one block per SM run
// the plane kernels as well, without a choice: they report 0, and writing that back changes nothing.
bool fused_selectable(int n, int prec);
int launch_planes_fwd(pgj_ctx* c, int loads, int mode, cudaStream_t s, cudaGraphConditionalHandle hif = 0);
int launch_planes_z(pgj_ctx* c, int loads, bool init, cudaStream_t s);
int launch_planes_inv(pgj_ctx* c, int loads, bool init, cudaStream_t s, cudaGraphConditionalHandle h, bool set_cond);
int launch_planes_shat(pgj_ctx* c, int loads, cudaStream_t s);
// z = P s G s P r of node-major FP64 vectors (FP64 contexts); r and z may be the same
int launch_planes_apply(pgj_ctx* c, int loads, const double* r, double* z, cudaStream_t s);
// copies the scale fields of the loads' designs by component, in the context precision (pgj_resident.cu)
int launch_scale_planes(pgj_ctx* c, int loads, cudaStream_t s);
// cluster-resident PCG (pgj_resident.cu): a whole attempt's recurrence in one launch
const ResidentKernel* resident_prepare(int n, int prec);
size_t resident_halo_bytes(int n, int prec);
int launch_resident(pgj_ctx* c, int loads, cudaStream_t s);
// The resident kernel runs the plain recurrences: the flexible direction update, FP64 arithmetic on FP32
// vectors and the refinement sweeps keep the separate kernels, as does a context set to step-by-step.
inline bool uses_resident(const pgj_ctx* c) {
  return c->res && c->four && !c->flex && !c->op64 && !(c->prec == PGJ_FP32 && c->mixed_mode == 1);
}
// pcg (pgj_pcg.cu)
int launch_update_ur(pgj_ctx* c, int loads, int prec, double* u64, void* uT, cudaStream_t s);
int launch_update_p(pgj_ctx* c, int loads, int prec, bool init, cudaStream_t s, cudaGraphConditionalHandle h,
                    bool set_cond);
int launch_init_mask(pgj_ctx* c, int loads, cudaStream_t s);
int launch_fold64(pgj_ctx* c, int loads, cudaStream_t s);
// mixed refinement (pgj_pcg.cu): inner residual r = T(r64), d = 0, inner targets and masks;
// then x += d for the loads solved in this sweep
int launch_inner_start(pgj_ctx* c, int loads, double inner_rtol, cudaStream_t s);
int launch_inner_finish(pgj_ctx* c, int loads, cudaStream_t s);
// reliable-update mixed solve (pgj_pcg.cu)
int launch_rel_start(pgj_ctx* c, int loads, cudaStream_t s);
int launch_decide(pgj_ctx* c, int loads, cudaGraphConditionalHandle h, cudaStream_t s);
int launch_rel_cond(pgj_ctx* c, int loads, cudaGraphConditionalHandle h, cudaStream_t s);
int launch_rel_fold(pgj_ctx* c, int loads, bool all, cudaStream_t s);
int launch_rel_sync(pgj_ctx* c, int loads, cudaStream_t s);
// energy (pgj_energy.cu)
int launch_energies(pgj_ctx* c, int loads, const double* u, const double* macros_dev, double* e, cudaStream_t s);
int launch_effective_tensor(pgj_ctx* c, const double* a, const double* u, double* C, cudaStream_t s);

// Points the context's per-design views (a, scale) at design d for the lifetime of the scope, so that the
// single-design scale build runs on it.
struct DesignScope {
  pgj_ctx* c;
  double* a;
  double* scale;
  DesignScope(pgj_ctx* ctx, int d);
  ~DesignScope();
};

int set_cuda_error(cudaError_t e);
// one-time kernel attributes (dynamic shared memory limits); called at context creation
int prepare_rows();
// the bounded waits of the OC updates (pgj_outer.cu) and the resident kernel, with nothing to complete them
int grid_wait_selftest(int limit_us, double* record, bool* expired, cudaStream_t s);
int launch_cluster_wait_selftest(int limit_us, int* flag, cudaStream_t s);
// times candidate tile shapes of the Green passes and keeps the fastest
int autotune_fft(pgj_ctx* c, cudaStream_t s);
int prepare_fft_kernels();
inline int check_launch() {
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? PGJ_OK : set_cuda_error(e);
}
}  // namespace pgj
