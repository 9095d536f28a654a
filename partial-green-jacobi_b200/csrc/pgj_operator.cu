// Right-hand side, norms, stiffness-diagonal scaling and projection, and the table of tile shapes. The
// operator itself is in pgj_rows.cuh.
#include "pgj_internal.h"
#include <cmath>
#include <cstdlib>

namespace pgj {

// Tile shapes of the Green passes per (grid edge, precision), picked offline by the project's tuner
// (partial-green-jacobi_b200/tune_tiles.py, which times every candidate on a B200 and writes
// pgj_tiles.inc). Contexts of a tabulated size take these shapes without timing anything, so the
// block decomposition, and with it the summation order of every block-partial reduction, is the
// same in every process, batch size and run. Sizes outside the table are tuned by timing at
// context creation (autotune_fft); PGJ_AUTOTUNE=1 forces timing for every size (that is how the
// table is made). The operator's shapes are computed (rows_geom).
static const TileEntry kTileTable[] = {
#include "pgj_tiles.inc"
    {0, 0, 0, 0, 0}};

bool tile_table(int n, int prec, TileEntry* out) {
  if (const char* e = std::getenv("PGJ_AUTOTUNE"))
    if (e[0] == '1') return false;
  for (const TileEntry& t : kTileTable)
    if (t.n == n && t.prec == prec) { *out = t; return true; }
  return false;
}

// --------------------------------------------------------------------------- right-hand side
// f(node) = -V sum over the 8 elements e = node - b of B_c(b)^T (a_e C0 eps), B_c the element-centre
// gradient (+-1/(4h) per axis); same arithmetic as hybrid_kernels.cu:50-68.
__global__ void k_rhs(int n, int loads, int lpd, const double* __restrict__ a, const double* __restrict__ macros,
                      double lam, double mu, double* __restrict__ f) {
  const size_t N = size_t(n) * n * n;
  const size_t node = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const int load = blockIdx.y;
  if (node >= N || load >= loads) return;
  a += size_t(load / lpd) * N;  // this load's design
  const int x = int(node % n), y = int((node / n) % n), z = int(node / (size_t(n) * n));
  const double* m = macros + 6 * load;
  // C0 eps (Voigt, engineering shear)
  const double tr = m[0] + m[1] + m[2];
  double s0[6];
  s0[0] = lam * tr + 2 * mu * m[0];
  s0[1] = lam * tr + 2 * mu * m[1];
  s0[2] = lam * tr + 2 * mu * m[2];
  s0[3] = mu * m[3]; s0[4] = mu * m[4]; s0[5] = mu * m[5];
  const double h = 1.0 / n, g = 1.0 / (4 * h), vol = h * h * h;
  double fx = 0, fy = 0, fz = 0;
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const int ex = wrapi(x - (b & 1), n), eyy = wrapi(y - ((b >> 1) & 1), n), ez = wrapi(z - ((b >> 2) & 1), n);
    const double ae = a[(size_t(ez) * n + eyy) * n + ex];
    const double dx = (b & 1) ? g : -g, dy = (b & 2) ? g : -g, dz = (b & 4) ? g : -g;
    double s[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) s[k] = ae * s0[k];
    fx -= vol * (dx * s[0] + dy * s[5] + dz * s[4]);
    fy -= vol * (dx * s[5] + dy * s[1] + dz * s[3]);
    fz -= vol * (dx * s[4] + dy * s[3] + dz * s[2]);
  }
  double* o = f + size_t(load) * 3 * N + 3 * node;
  o[0] = fx; o[1] = fy; o[2] = fz;
}

int launch_rhs(pgj_ctx* c, int loads, const double* macros_dev, double* f, cudaStream_t s) {
  const size_t N = size_t(c->N);
  dim3 grid(unsigned((N + 255) / 256), loads);
  k_rhs<<<grid, 256, 0, s>>>(c->n, loads, c->lpd, c->a, macros_dev, c->lam, c->mu, f);
  return check_launch();
}

// --------------------------------------------------------------------------- norms / targets
// ||f|| per load, target^2 = max(rtol ||f||, 1e-13/sqrt(n))^2; resets iteration counters and
// latches (resident.py:187-191).
__global__ void k_norms(int n, const double* __restrict__ f, double rtol, LoadScalars* scal, double* partials) {
  const size_t N3 = 3 * size_t(n) * n * n;
  const int load = blockIdx.y;
  const double* fl = f + size_t(load) * N3;
  double acc[1] = {0.0};
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < N3; i += size_t(gridDim.x) * blockDim.x) {
    const double v = fl[i];
    acc[0] += v * v;
  }
  __shared__ double red[32];
  block_sum<1>(acc, red);
  double* part = partials + size_t(load) * kPartialQ * kMaxPartials;
  if (threadIdx.x == 0) part[blockIdx.x] = acc[0];
  LoadScalars& S = scal[load];
  if (!last_block(&S.ticket[kTicketAux], gridDim.x)) return;
  if (threadIdx.x < 32) {
    const double s2 = warp_sum_partials(part, gridDim.x);
    if (threadIdx.x == 0) {
      const double norm = sqrt(s2);
      const double t = fmax(norm * rtol, 1e-13 / sqrt(double(n)));
      S.norm = norm;
      S.target2 = t * t;
      S.iterations = 0;
      S.total_iterations = 0;
      S.touched = 0;
      S.bad = 0;
      S.failed = 0;
      S.active = 0;
      S.frozen = 0;
      S.restarts = 0;
    }
  }
}

int launch_norms(pgj_ctx* c, int loads, const double* f, double rtol, cudaStream_t s) {
  dim3 grid(148, loads);
  k_norms<<<grid, 256, 0, s>>>(c->n, f, rtol, c->scal, c->partials);
  return check_launch();
}

// --------------------------------------------------------------------------- projection of u
// mean over nodes per component, then subtract (certification projection, resident.py:133-134).
__global__ void k_mean3(int n, const double* __restrict__ u, int which, LoadScalars* scal, double* partials) {
  const size_t N = size_t(n) * n * n;
  const int load = blockIdx.y;
  if (which == 0 && scal[load].frozen) return;  // certification of a design that took its last attempt
  LoadScalars& S = scal[load];
  grid_mean3(N, u + size_t(load) * 3 * N, which ? S.mean_r : S.mean_u, S, partials + size_t(load) * kPartialQ * kMaxPartials);
}

__global__ void k_sub_mean3(int n, double* __restrict__ u, const LoadScalars* scal) {
  const size_t N3 = 3 * size_t(n) * n * n;
  const int load = blockIdx.y;
  if (scal[load].frozen) return;
  double* ul = u + size_t(load) * N3;
  const double m0 = scal[load].mean_u[0], m1 = scal[load].mean_u[1], m2 = scal[load].mean_u[2];
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < N3; i += size_t(gridDim.x) * blockDim.x) {
    const int c = int(i % 3);
    ul[i] -= (c == 0 ? m0 : (c == 1 ? m1 : m2));
  }
}

int launch_mean3(pgj_ctx* c, int loads, const double* v, int which, cudaStream_t s) {
  dim3 grid(148, loads);
  k_mean3<<<grid, 256, 0, s>>>(c->n, v, which, c->scal, c->partials);
  return check_launch();
}

int launch_project_u(pgj_ctx* c, int loads, double* u, cudaStream_t s) {
  int st = launch_mean3(c, loads, u, 0, s);
  if (st) return st;
  dim3 grid2(296, loads);
  k_sub_mean3<<<grid2, 256, 0, s>>>(c->n, u, c->scal);
  return check_launch();
}

// --------------------------------------------------------------------------- diagonal scaling
// log d(node, c), d = sum_b a(node - b) diag(Ke)[b][c]; partial sums of log d for the mean.
__global__ void k_logdiag(int n, const double* __restrict__ a, const double* __restrict__ ed, double* __restrict__ out,
                          LoadScalars* scal, double* partials) {
  const size_t N = size_t(n) * n * n;
  double acc[1] = {0.0};
  for (size_t node = size_t(blockIdx.x) * blockDim.x + threadIdx.x; node < N; node += size_t(gridDim.x) * blockDim.x) {
    const int x = int(node % n), y = int((node / n) % n), z = int(node / (size_t(n) * n));
    double d[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const int ex = wrapi(x - (b & 1), n), eyy = wrapi(y - ((b >> 1) & 1), n), ez = wrapi(z - ((b >> 2) & 1), n);
      const double ae = a[(size_t(ez) * n + eyy) * n + ex];
#pragma unroll
      for (int c = 0; c < 3; ++c) d[c] += ae * ed[3 * b + c];
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double q = log(d[c]);
      out[3 * node + c] = q;
      acc[0] += q;
    }
  }
  __shared__ double red[32];
  block_sum<1>(acc, red);
  if (threadIdx.x == 0) partials[blockIdx.x] = acc[0];
  if (!last_block(&scal[0].ticket[kTicketAux2], gridDim.x)) return;
  if (threadIdx.x < 32) {
    const double s2 = warp_sum_partials(partials, gridDim.x);
    if (threadIdx.x == 0) partials[kMaxPartials - 1] = s2 / double(3 * N);
  }
}

__global__ void k_exp_scale(size_t count, double* __restrict__ q, const double* __restrict__ mean, double coef) {
  const double m = *mean;
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += size_t(gridDim.x) * blockDim.x)
    q[i] = exp(coef * (q[i] - m));
}

__global__ void k_fill(size_t count, double* __restrict__ q, double v) {
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += size_t(gridDim.x) * blockDim.x) q[i] = v;
}

// diag(Ke) per local node b (bit order), 2x2x2 Gauss, isotropic C0; host-side constant.
void element_diagonal(int n, double lam, double mu, double* ed) {
  const double g = 1.0 / std::sqrt(3.0);
  for (int i = 0; i < 24; ++i) ed[i] = 0.0;
  for (int q = 0; q < 8; ++q) {
    const double p[3] = {0.5 + ((q & 1) ? 0.5 : -0.5) * g, 0.5 + ((q & 2) ? 0.5 : -0.5) * g,
                         0.5 + ((q & 4) ? 0.5 : -0.5) * g};
    for (int b = 0; b < 8; ++b) {
      const int v[3] = {b & 1, (b >> 1) & 1, (b >> 2) & 1};
      double fac[3], grad[3];
      for (int d = 0; d < 3; ++d) fac[d] = v[d] ? p[d] : 1 - p[d];
      for (int d = 0; d < 3; ++d) {
        double prod = 1.0;
        for (int e = 0; e < 3; ++e) if (e != d) prod *= fac[e];
        grad[d] = (2 * v[d] - 1) * prod * n;
      }
      // diagonal of B^T C B for the x, y, z dofs of node b
      const double l2m = lam + 2 * mu;
      ed[3 * b + 0] += l2m * grad[0] * grad[0] + mu * (grad[1] * grad[1] + grad[2] * grad[2]);
      ed[3 * b + 1] += l2m * grad[1] * grad[1] + mu * (grad[0] * grad[0] + grad[2] * grad[2]);
      ed[3 * b + 2] += l2m * grad[2] * grad[2] + mu * (grad[0] * grad[0] + grad[1] * grad[1]);
    }
  }
  const double vol8 = 1.0 / (double(n) * n * n) / 8.0;
  for (int i = 0; i < 24; ++i) ed[i] *= vol8;
}

int launch_scale(pgj_ctx* c, double alpha, cudaStream_t s) {
  const size_t count = 3 * size_t(c->N);
  if (alpha == 0.0) {
    k_fill<<<296, 256, 0, s>>>(count, c->scale, 1.0);
    return check_launch();
  }
  double* edd = c->aux;  // 24 diagonal entries, staged once in the context's aux block
  if (!c->diag_staged) {
    double ed[24];
    element_diagonal(c->n, c->lam, c->mu, ed);
    cudaError_t e = cudaMemcpyAsync(edd, ed, sizeof(ed), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return set_cuda_error(e);
    c->diag_staged = 1;
  }
  k_logdiag<<<296, 256, 0, s>>>(c->n, c->a, edd, c->scale, c->scal, c->aux + kAuxPartials);
  int st = check_launch();
  if (st) return st;
  k_exp_scale<<<296, 256, 0, s>>>(count, c->scale, c->aux + kAuxPartials + kMaxPartials - 1, -0.5 * alpha);
  return check_launch();
}

}  // namespace pgj
