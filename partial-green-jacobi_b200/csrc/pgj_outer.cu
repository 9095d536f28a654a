// Design-update chains kept on the device: density filters, projection + SIMP, and the optimality
// criteria (OC) volume bisection.
//
// Study II (paper conventions, exp/asg_sctop_reproduction_20261105/outer.cu:8-39 and
// reproduction.py:69-118): clipped cone filter, tanh(beta, eta) projection, damped OC
// x' = clip(x max(1e-10, ratio/mid)^exponent, max(floor, x-move), min(1, x+move)), MATLAB
// bisection stop (hi-lo)/(hi+lo) <= 1e-4, at most 180 steps.
// Study I (exp/asg_gpu_resident_20261103/outer.cu:7-37, outer.py:26-44): periodic separable
// Gaussian (scipy.ndimage correlation order), tanh projection at 1/2, SIMP eta=1e-4, 45 steps.
//
// A bisection is a serial chain of 45 to 163 steps with two or three grid-wide dependencies each around
// a few microseconds of work. Both updates therefore run as one cooperative launch whose blocks keep
// the bounds in registers and meet at a bounded grid barrier; every block forms the volume from the
// same partial sums in the same order and so takes the same branch. (As separate launches, 180 steps
// were always issued, three launches each, most of them after the bisection had stopped. Paper update 4.5 ms
// against 1.5 ms at n = 64 and 2.8 against 0.85 at n = 16; Study I update 1.2 against 0.42 ms at n = 32,
// 6.9 against 2.3 at n = 96.)
#include "pgj_internal.h"
#include <algorithm>
#include <cmath>
#include <cstring>

namespace pgj {

// --------------------------------------------------------------------------- grid barrier
// Barrier over the blocks of a cooperative launch: one counter that only grows. Bounded: a block that
// waits longer than kGridWaitNs (other work can hold SMs that later blocks of the grid still need)
// marks the record dead, and every block leaves at its next barrier.
struct GridBar {
  unsigned count;
  int dead;
};
constexpr unsigned long long kGridWaitNs = 20000000000ull;

__device__ __forceinline__ bool grid_barrier(GridBar* b, unsigned& target, unsigned long long limit = kGridWaitNs) {
  target += gridDim.x;
  __syncthreads();
  int dead = 0;
  if (flat_tid() == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&b->count) : "memory");
    unsigned long long t0 = 0, t = 0;
    for (unsigned tries = 0; tries < 0x7fffffffu; ++tries) {
      unsigned c;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(&b->count) : "memory");
      if (c >= target) break;
      if ((tries & 255u) == 255u) {
        dead = *(volatile int*)&b->dead;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
        if (t0 == 0) t0 = t;
        if (dead || t - t0 > limit) {
          dead = 1;
          *(volatile int*)&b->dead = 1;
          break;
        }
      }
    }
  }
  return __syncthreads_or(dead) == 0;
}

// Leaves the mark of an update that gave up in the record a caller without a synchronisation reads: -1 steps and a
// NaN change. grid_max takes the largest bit pattern, which keeps the NaN whatever other blocks still add.
__device__ __forceinline__ void oc_gave_up(double* bounds) {
  if (flat_tid() != 0) return;
  *(volatile double*)(bounds + 3) = -1.0;
  atomicMax(reinterpret_cast<unsigned long long*>(bounds + 4), 0x7ff8000000000000ull);
}

// Self-test: a barrier that needs one more arrival than there are blocks.
__global__ void k_grid_wait_selftest(GridBar* bar, double* bounds, unsigned long long limit) {
  unsigned target = 1;
  if (!grid_barrier(bar, target, limit)) oc_gave_up(bounds);
}

// --------------------------------------------------------------------------- cone filter
// Clipped cone filter y(p) = sum_j w_j x(p + d_j) over the taps whose neighbour lies inside the grid
// (no periodic wrap), taps summed in table order with one fused multiply-add each (the order of the
// reference's loop), so the result does not depend on the tiling.
//
// Taps within kConeR cells: a block of 32 x 8 threads (x fastest) takes a tile of 32 x 8 x kConeZ cells.
// The tile and its halo sit in shared memory, zero outside the grid (a tap that falls there adds zero),
// and a thread sums kConeZ cells along z at once: one broadcast read of a tap, then kConeZ reads and
// multiply-adds without bounds tests. Table and tile stay within the 48 KB that a kernel has without setting
// a limit (384 taps hold every offset of the radius). Reads of the tile bound it: 14.7 us a call at n = 64 with 93 taps
// (31.3 at n = 96), against 35.2 (76.4) with the neighbours read from global memory one by one.
//
// Farther or longer tables take the general loop, which reads neighbours through the L1, 1, 2 or 4 cells along z per
// thread, kConeTaps taps at a time. Instructions bound it on large grids (tests, addresses and selects of a tap are
// shared by a thread's cells), the latency of a group's loads on small ones. us a call, one cell per thread with a branch
// per tap / four cells one after the other / this loop: 389 taps n = 24 54 / 217 / 35, 64 123 / 281 / 103, 128 647 /
// 1403 / 543; 4139 taps n = 24 539 / 2235 / 330, 64 1165 / 2710 / 1026.
constexpr int kConeX = 32, kConeY = 8, kConeZ = 4, kConeR = 3, kConeTaps = 384;
struct alignas(16) ConeTap {
  double w;
  long long lin;  // offset of the neighbour in the tile or in the field
};
struct alignas(16) ConeWide {
  int dx, dy, dz, pad;
  long long lin;
  double w;
};
constexpr int kConeTile = (kConeX + 2 * kConeR) * (kConeY + 2 * kConeR) * (kConeZ + 2 * kConeR);
union ConeSmem {
  struct {
    ConeTap taps[kConeTaps];
    double tile[kConeTile];
  };
  ConeWide wide[kConeTaps];
};

// Radius of the tap table (max |offset|) if it fits the tile form, else -1; the tile form's tap table is
// then staged in `sm`. Called by every thread of a 32 x 8 block. A weight that is not finite does not fit: a tap
// that falls outside the grid would not add zero.
__device__ __forceinline__ int cone_stage(ConeSmem& sm, const int32_t* __restrict__ offsets,
                                          const double* __restrict__ weights, int count) {
  const int tid = flat_tid();
  if (count > kConeTaps) return -1;
  __shared__ int radius;
  if (tid == 0) radius = 0;
  __syncthreads();
  int r = 0;
  for (int j = tid; j < 3 * count; j += kConeX * kConeY) {
    const int d = offsets[j];
    r = max(r, d < -kConeR || d > kConeR ? kConeR + 1 : abs(d));
  }
  for (int j = tid; j < count; j += kConeX * kConeY)
    if (!isfinite(weights[j])) r = kConeR + 1;
  atomicMax(&radius, r);
  __syncthreads();
  r = radius;
  if (r > kConeR) return -1;
  const int px = kConeX + 2 * r, py = kConeY + 2 * r;
  for (int j = tid; j < count; j += kConeX * kConeY) {
    sm.taps[j].w = weights[j];
    sm.taps[j].lin = (offsets[3 * j + 2] * py + offsets[3 * j + 1]) * px + offsets[3 * j];
  }
  __syncthreads();
  return r;
}

// Tiles of `depth` planes along z.
__host__ __device__ inline int cone_tiles(int n, int depth) {
  return ((n + kConeX - 1) / kConeX) * ((n + kConeY - 1) / kConeY) * ((n + depth - 1) / depth);
}

// General loop over tile `t` (tiles x fastest, then y, then z) of K planes, K cells along z per thread: any table, taps
// outside the grid skipped. The cells share a tap's reads and its tests in the plane, and the loads of U taps are in
// flight together, without branches: where a tap falls outside, a cell of the thread's own stands in and the sum is left
// as it was.
template <int K, class Out>
__device__ __forceinline__ void cone_general(ConeSmem& sm, int n, const int32_t* __restrict__ offsets,
                                             const double* __restrict__ weights, int count, int t, const double* src,
                                             Out out) {
  const int nx = (n + kConeX - 1) / kConeX, ny = (n + kConeY - 1) / kConeY;
  const int bz = t / (nx * ny), rem = t - bz * nx * ny, by = rem / nx, bx = rem - by * nx;
  const int cx = bx * kConeX + threadIdx.x, cy = by * kConeY + threadIdx.y, cz = bz * K;
  constexpr int U = K == 4 ? 2 : 4;
  static_assert(kConeTaps % U == 0, "chunks are whole groups");
  const bool inside = cx < n && cy < n;
  const unsigned un = unsigned(n);
  const size_t plane = size_t(n) * n;
  const size_t at0 = (size_t(cz) * n + cy) * n + cx;
  const double* cell = src + at0;
  double acc[K];
#pragma unroll
  for (int k = 0; k < K; ++k) acc[k] = 0.0;
  for (int first = 0; first < count; first += kConeTaps) {
    const int m = min(kConeTaps, count - first), groups = (m + U - 1) / U;
    __syncthreads();  // the previous chunk has been read
    for (int j = flat_tid(); j < groups * U; j += kConeX * kConeY) {
      ConeWide w = {n, n, n, 0, 0, 0.0};  // fills up the last group: outside from any cell
      if (j < m) {
        const int at = 3 * (first + j);
        w.dx = offsets[at]; w.dy = offsets[at + 1]; w.dz = offsets[at + 2];
        w.lin = (static_cast<long long>(w.dz) * n + w.dy) * n + w.dx;
        w.w = weights[first + j];
      }
      sm.wide[j] = w;
    }
    __syncthreads();
    if (!inside) continue;
#pragma unroll 1
    for (int g = 0; g < groups; ++g) {
      double w[U], v[U][K];
      bool in[U][K];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const ConeWide& tap = sm.wide[g * U + u];
        w[u] = tap.w;
        const bool xy = unsigned(cx) + unsigned(tap.dx) < un && unsigned(cy) + unsigned(tap.dy) < un;
#pragma unroll
        for (int k = 0; k < K; ++k) {
          in[u][k] = xy && unsigned(cz + k) + unsigned(tap.dz) < un;
          v[u][k] = cell[in[u][k] ? tap.lin + static_cast<long long>(k * plane) : 0];
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int k = 0; k < K; ++k)
          acc[k] = in[u][k] ? fma(w[u], v[u][k], acc[k]) : acc[k];
    }
  }
  if (inside)
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (cz + k < n) out(at0 + k * plane, acc[k]);
}

// Tiled form over tile `t` of kConeZ planes; out(cell, value) receives the cells.
template <class Out>
__device__ __forceinline__ void cone_tile(ConeSmem& sm, int radius, int n, int count, int t, const double* src, Out out) {
  const int nx = (n + kConeX - 1) / kConeX, ny = (n + kConeY - 1) / kConeY;
  const int bz = t / (nx * ny), rem = t - bz * nx * ny, by = rem / nx, bx = rem - by * nx;
  const int lx = threadIdx.x, ly = threadIdx.y;
  const int x0 = bx * kConeX, y0 = by * kConeY, z0 = bz * kConeZ;
  const int cx = x0 + lx, cy = y0 + ly;
  double acc[kConeZ];
#pragma unroll
  for (int k = 0; k < kConeZ; ++k) acc[k] = 0.0;
  const int px = kConeX + 2 * radius, py = kConeY + 2 * radius, pz = kConeZ + 2 * radius;
  __syncthreads();  // the previous tile has been read
  // a thread fills whole z columns of the tile, all loads of a column in flight together
  for (int p = flat_tid(); p < px * py; p += kConeX * kConeY) {
    const int y = p / px, x = p - y * px, gx = x0 + x - radius, gy = y0 + y - radius;
    const bool in = unsigned(gx) < unsigned(n) && unsigned(gy) < unsigned(n);
    double v[kConeZ + 2 * kConeR];
#pragma unroll
    for (int z = 0; z < kConeZ + 2 * kConeR; ++z) {
      const int gz = z0 + z - radius;
      v[z] = in && z < pz && unsigned(gz) < unsigned(n) ? __ldcg(src + (size_t(gz) * n + gy) * n + gx) : 0.0;
    }
#pragma unroll
    for (int z = 0; z < kConeZ + 2 * kConeR; ++z)
      if (z < pz) sm.tile[z * px * py + p] = v[z];
  }
  __syncthreads();
  const double* at = sm.tile + (radius * py + ly + radius) * px + lx + radius;
  const int pl = px * py;
  // eight taps' reads are in flight before their multiply-adds (a tap at a time waits out two shared
  // memory latencies per tap)
  constexpr int U = 8;
  int j = 0;
  for (; j + U <= count; j += U) {
    double w[U], v[U][kConeZ];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const ConeTap tap = sm.taps[j + u];
      w[u] = tap.w;
      const double* p = at + int(tap.lin);
#pragma unroll
      for (int k = 0; k < kConeZ; ++k) v[u][k] = p[k * pl];
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int k = 0; k < kConeZ; ++k) acc[k] += w[u] * v[u][k];
  }
  for (; j < count; ++j) {
    const double w = sm.taps[j].w;
    const double* p = at + int(sm.taps[j].lin);
#pragma unroll
    for (int k = 0; k < kConeZ; ++k) acc[k] += w * p[k * pl];
  }
  if (cx < n && cy < n)
#pragma unroll
    for (int k = 0; k < kConeZ; ++k)
      if (z0 + k < n) out((size_t(z0 + k) * n + cy) * n + cx, acc[k]);
}

// Calls body(filter) for every tile of the block; filter(src, out) filters the tile of the field `src`, out(cell, value)
// receives its cells.
template <class Body>
__device__ __forceinline__ void cone_fields(ConeSmem& sm, int radius, int n, const int32_t* __restrict__ offsets,
                                            const double* __restrict__ weights, int count, Body body) {
  const int t = blockIdx.x, nblk = gridDim.x;
  if (radius >= 0) {
    for (int i = t; i < cone_tiles(n, kConeZ); i += nblk)
      body([&](const double* src, auto out) { cone_tile(sm, radius, n, count, i, src, out); });
  } else if (cone_tiles(n, 1) <= nblk) {  // as few planes a tile as give every block one
    if (t < cone_tiles(n, 1))
      body([&](const double* src, auto out) { cone_general<1>(sm, n, offsets, weights, count, t, src, out); });
  } else if (cone_tiles(n, 2) <= nblk) {
    if (t < cone_tiles(n, 2))
      body([&](const double* src, auto out) { cone_general<2>(sm, n, offsets, weights, count, t, src, out); });
  } else {
    for (int i = t; i < cone_tiles(n, kConeZ); i += nblk)
      body([&](const double* src, auto out) { cone_general<kConeZ>(sm, n, offsets, weights, count, i, src, out); });
  }
}

__global__ void __launch_bounds__(kConeX * kConeY) k_cone_filter(int n, const int32_t* __restrict__ offsets,
                                                                 const double* __restrict__ weights, int count,
                                                                 const double* __restrict__ x, double* __restrict__ y) {
  extern __shared__ __align__(16) unsigned char raw[];
  ConeSmem& sm = *reinterpret_cast<ConeSmem*>(raw);
  const int radius = cone_stage(sm, offsets, weights, count);
  cone_fields(sm, radius, n, offsets, weights, count,
              [&](auto filter) { filter(x, [&](size_t i, double v) { y[i] = v; }); });
}

// te = tanh(beta eta), den = te + tanh(beta (1 - eta))
__device__ __forceinline__ void paper_phys(double t, double hs, double beta, double eta, double emin, double te,
                                           double den, double& ph, double& dp, double& a) {
  const double q = tanh(beta * (t / hs - eta));
  const double rho = (te + q) / den;
  ph = rho;
  dp = beta * (1 - q * q) / den;
  a = emin + (1 - emin) * rho * rho * rho;
}

__global__ void k_paper_project(size_t N, const double* __restrict__ t, const double* __restrict__ hs, double beta,
                                double eta, double emin, double* __restrict__ ph, double* __restrict__ dp,
                                double* __restrict__ a) {
  const double te = tanh(beta * eta), den = te + tanh(beta * (1 - eta));
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < N; i += size_t(gridDim.x) * blockDim.x) {
    double p, d, aa;
    paper_phys(t[i], hs[i], beta, eta, emin, te, den, p, d, aa);
    ph[i] = p; dp[i] = d; a[i] = aa;
  }
}

// Bisection record shared with the callers: lo, hi, continue flag, steps taken, max |xnew - x|.
struct OCArgs {
  int n;
  const int32_t* offsets;  // paper: cone taps
  const double* weights;   // cone weights, or the Gaussian's 2 radius + 1
  int count;               // taps, or the Gaussian's radius
  const double *x, *ph, *dp, *hs, *energy;
  double volume, beta, eta, emin, move, exponent, floor_;
  double* xnew;
  double *f0, *f1, *f2, *f3;  // ratio, dv (both left to the caller: g = -ratio dv), temporaries
  double* bounds;
  GridBar* bar;
  double* partials;
};

// Sum of one partial per block, in block order, by every warp of the block (all threads get the value).
__device__ __forceinline__ double sum_partials(const double* p) {
  const int lane = flat_tid() & 31;
  double s = 0.0;
  for (int i = lane; i < int(gridDim.x); i += 32) s += __ldcg(p + i);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// max over the grid of a non-negative value, into a record that starts at zero (bit patterns of
// non-negative doubles are ordered like the values); NaN leaves it, as fmax does
__device__ __forceinline__ void grid_max(double m, double* out) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((flat_tid() & 31) == 0 && m > 0.0)
    atomicMax(reinterpret_cast<unsigned long long*>(out), static_cast<unsigned long long>(__double_as_longlong(m)));
}

// Fields that other blocks wrote are read after a grid barrier only, whose acquire orders plain loads too.
//
// Damped OC update of the paper's chain (reproduction.py:92-118): filtered sensitivities, ratio, and the
// bisection of the multiplier. Per step: candidate design; barrier; cone filter of it, projection, volume
// partials; barrier.
__global__ void __launch_bounds__(kConeX * kConeY) k_paper_oc(const OCArgs A) {
  extern __shared__ __align__(16) unsigned char raw[];
  ConeSmem& sm = *reinterpret_cast<ConeSmem*>(raw);
  __shared__ double red[32];
  const int n = A.n, tid = flat_tid();
  const size_t N = size_t(n) * n * n, stride = size_t(gridDim.x) * (kConeX * kConeY);
  const size_t first = size_t(blockIdx.x) * (kConeX * kConeY) + tid;
  const int radius = cone_stage(sm, A.offsets, A.weights, A.count);
  unsigned target = 0;
  // g = dp 3 (1 - emin) ph^2 energy / hs and v = dp / hs, filtered; ratio = -(g / N) / dv
  for (size_t i = first; i < N; i += stride) {
    const double dp = A.dp[i], ph = A.ph[i], hs = A.hs[i];
    A.f2[i] = dp * (3 * (1 - A.emin) * (ph * ph)) * A.energy[i] / hs;
    A.f3[i] = dp / hs;
  }
  if (!grid_barrier(A.bar, target)) return oc_gave_up(A.bounds);
  const double dN = double(N);
  cone_fields(sm, radius, n, A.offsets, A.weights, A.count, [&](auto filter) {
    filter(A.f2, [&](size_t i, double v) { A.f0[i] = v; });
    filter(A.f3, [&](size_t i, double v) {
      A.f0[i] = -(A.f0[i] / dN) / v;
      A.f1[i] = v;
    });
  });
  if (!grid_barrier(A.bar, target)) return oc_gave_up(A.bounds);
  const double te = tanh(A.beta * A.eta), den = te + tanh(A.beta * (1 - A.eta));
  double lo = 0.0, hi = 1e9, steps = 0.0;
  bool go = true;
  for (int it = 0; it < 180 && go; ++it) {
    const double mid = 0.5 * (lo + hi);
    for (size_t i = first; i < N; i += stride) {
      const double xi = A.x[i];
      const double v = xi * pow(fmax(1e-10, __ldcg(A.f0 + i) / mid), A.exponent);
      A.xnew[i] = fmax(A.floor_, fmax(xi - A.move, fmin(1.0, fmin(xi + A.move, v))));
    }
    if (!grid_barrier(A.bar, target)) return oc_gave_up(A.bounds);
    double acc[1] = {0.0};
    cone_fields(sm, radius, n, A.offsets, A.weights, A.count, [&](auto filter) {
      filter(A.xnew, [&](size_t i, double v) {
        double p, d, a;
        paper_phys(v, A.hs[i], A.beta, A.eta, A.emin, te, den, p, d, a);
        acc[0] += p;
      });
    });
    block_sum<1>(acc, red);
    if (tid == 0) A.partials[blockIdx.x] = acc[0];
    if (!grid_barrier(A.bar, target)) return oc_gave_up(A.bounds);
    const double vol = sum_partials(A.partials) / dN;
    if (vol > A.volume) lo = mid; else hi = mid;
    steps += 1.0;
    go = (hi - lo) / (hi + lo) > 1e-4 && hi > 1e-40;
  }
  double m = 0.0;
  for (size_t i = first; i < N; i += stride) m = fmax(m, fabs(__ldcg(A.xnew + i) - A.x[i]));
  grid_max(m, A.bounds + 4);
  if (blockIdx.x == 0 && tid == 0 && !*(volatile int*)&A.bar->dead) {
    A.bounds[0] = lo;
    A.bounds[1] = hi;
    A.bounds[2] = go ? 1.0 : 0.0;
    A.bounds[3] = steps;
  }
}

// max |a - b| (single block reduction into out[0])
__global__ void k_absmax_diff(size_t N, const double* __restrict__ a, const double* __restrict__ b, double* out) {
  double m = 0.0;
  for (size_t i = threadIdx.x; i < N; i += blockDim.x) m = fmax(m, fabs(a[i] - b[i]));
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
  __shared__ double red[32];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 32) {
    m = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
    if (threadIdx.x == 0) out[0] = m;
  }
}

// --------------------------------------------------------------------------- Study I
// y[i] = w[r] x[i] + sum_k w[r+k] (x[i-k] + x[i+k]) along one periodic axis.
__global__ void k_gauss_axis(int n, int axis, const double* __restrict__ w, int radius, const double* __restrict__ x,
                             double* __restrict__ y) {
  const size_t N = size_t(n) * n * n;
  const size_t stride = axis == 0 ? size_t(n) * n : (axis == 1 ? size_t(n) : 1);
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < N; i += size_t(gridDim.x) * blockDim.x) {
    const int coord = int((i / stride) % n);
    double v = w[radius] * x[i];
    for (int k = 1; k <= radius; ++k) {
      int lo = (coord - k) % n;
      if (lo < 0) lo += n;
      const int hi = (coord + k) % n;
      v += w[radius + k] * (x[i + (long long)(lo - coord) * (long long)stride] + x[i + (long long)(hi - coord) * (long long)stride]);
    }
    y[i] = v;
  }
}

__device__ __forceinline__ void s1_phys(double t, double b, double& p, double& d, double& a) {
  const double half = tanh(0.5 * b), q = tanh(b * (t - 0.5));
  p = (half + q) / (2 * half);
  d = b * (1 - q * q) / (2 * half);
  a = 1e-4 + (1.0 - 1e-4) * p * p * p;
}

__global__ void k_s1_project(size_t N, const double* __restrict__ t, double beta, double* __restrict__ ph,
                             double* __restrict__ dp, double* __restrict__ a) {
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < N; i += size_t(gridDim.x) * blockDim.x) {
    double p, d, aa;
    s1_phys(t[i], beta, p, d, aa);
    ph[i] = p; dp[i] = d; a[i] = aa;
  }
}

__global__ void k_s1_sens_in(size_t N, const double* __restrict__ ph, const double* __restrict__ dp,
                             const double* __restrict__ energy, double* __restrict__ gin) {
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < N; i += size_t(gridDim.x) * blockDim.x)
    gin[i] = dp[i] * 3 * (1. - 1e-4) * (ph[i] * ph[i]) * energy[i];
}

// ratio = max(g,1e-30)/max(dv,1e-30) in place; hi bound = max(ratio) * 1e4 (single-block max)
__global__ void k_s1_ratio(size_t N, double* __restrict__ g, const double* __restrict__ dv, double* bounds) {
  double m = 0.0;
  for (size_t i = threadIdx.x; i < N; i += blockDim.x) {
    const double r = fmax(g[i], 1e-30) / fmax(dv[i], 1e-30);
    g[i] = r;
    m = fmax(m, r);
  }
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
  __shared__ double red[32];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 32) {
    m = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
    if (threadIdx.x == 0) { bounds[0] = 0.0; bounds[1] = m * 1e4; bounds[2] = 1.0; bounds[3] = 0.0; }
  }
}

__global__ void k_s1_candidate(size_t N, const double* __restrict__ x, const double* __restrict__ ratio,
                               const double* bounds, double move, double* __restrict__ y) {
  const double lam = fmax((bounds[0] + bounds[1]) * 0.5, 1e-30);
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < N; i += size_t(gridDim.x) * blockDim.x) {
    const double lo = fmax(0., x[i] - move), hi = fmin(1., x[i] + move);
    y[i] = fmin(hi, fmax(lo, x[i] * sqrt(ratio[i] / lam)));
  }
}

__global__ void k_s1_volume(size_t N, const double* __restrict__ t, double beta, double target, double* bounds,
                            double* partials, int* ticket) {
  double acc[1] = {0.0};
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < N; i += size_t(gridDim.x) * blockDim.x) {
    double p, d, a;
    s1_phys(t[i], beta, p, d, a);
    acc[0] += p;
  }
  __shared__ double red[32];
  block_sum<1>(acc, red);
  if (threadIdx.x == 0) partials[blockIdx.x] = acc[0];
  if (!last_block(ticket, gridDim.x)) return;
  if (threadIdx.x < 32) {
    const double s = warp_sum_partials(partials, gridDim.x);
    if (threadIdx.x == 0) {
      const double mid = (bounds[0] + bounds[1]) * 0.5;
      if (s / double(N) > target) bounds[0] = mid; else bounds[1] = mid;
      bounds[3] += 1.0;
    }
  }
}

// Study I update (exp/asg_gpu_resident_20261103/outer.py:26-44) in one launch. A separable pass over z
// takes 32 neighbouring columns in shared memory (the candidate design is formed as the columns are
// read); the passes over y and x take kS1Rows rows of a plane with their y halo, one warp per row, so a
// row's x pass needs no block barrier. Per step: z pass; barrier; y and x passes, projection, volume
// partials; barrier. Each cell's sum runs in the order of the separate kernels.
constexpr int kS1Rows = 8, kS1Threads = 32 * kS1Rows;

// z pass over 32 columns: dst = filter of fin(cell, ld(cell)); four cells' loads are in flight together
template <class Ld, class Fin>
__device__ __forceinline__ void s1_columns(double* col, const double* w, int radius, int n, int tile, Ld ld, Fin fin,
                                           double* __restrict__ dst) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nn = n * n, c = tile * 32 + lane;
  const bool on = c < nn;
  using V = decltype(ld(size_t(0)));
  __syncthreads();  // the previous columns have been read
  for (int zb = warp; zb < n; zb += 4 * kS1Rows) {
    V v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (on && zb + u * kS1Rows < n) v[u] = ld(size_t(zb + u * kS1Rows) * nn + c);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (on && zb + u * kS1Rows < n)
        col[(zb + u * kS1Rows) * 32 + lane] = fin(size_t(zb + u * kS1Rows) * nn + c, v[u]);
  }
  __syncthreads();
  if (!on) return;
  for (int z = warp; z < n; z += kS1Rows) {
    double v = w[0] * col[z * 32 + lane];
    int lo = z, hi = z;
    for (int k = 1; k <= radius; ++k) {
      lo = lo == 0 ? n - 1 : lo - 1;
      hi = hi + 1 == n ? 0 : hi + 1;
      v += w[k] * (col[lo * 32 + lane] + col[hi * 32 + lane]);
    }
    dst[size_t(z) * nn + c] = v;
  }
}

// y and x passes over kS1Rows rows of one plane: out(cell, value)
template <class Out>
__device__ __forceinline__ void s1_rows(double* rows, const double* w, int radius, int n, int task,
                                        const double* src, Out out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int chunks = (n + kS1Rows - 1) / kS1Rows, z = task / chunks, y0 = (task - z * chunks) * kS1Rows;
  const int span = kS1Rows + 2 * radius;
  double* mid = rows + size_t(span) * n;
  const double* plane = src + size_t(z) * n * n;
  __syncthreads();  // the previous rows have been read
  batched_copy<8>(threadIdx.x, kS1Threads, span * n, [&](int e) {
    const int j = e / n, x = e - j * n;
    int y = (y0 - radius + j) % n;
    if (y < 0) y += n;
    return __ldcg(plane + y * n + x);
  }, [&](int e, double v) { rows[e] = v; });
  __syncthreads();
  const int y = y0 + warp;
  if (y >= n) return;
  const double* centre = rows + (warp + radius) * n;
  double* m = mid + warp * n;
  for (int x = lane; x < n; x += 32) {
    double v = w[0] * centre[x];
    for (int k = 1; k <= radius; ++k) v += w[k] * (centre[x - k * n] + centre[x + k * n]);
    m[x] = v;
  }
  __syncwarp();
  for (int x = lane; x < n; x += 32) {
    double v = w[0] * m[x];
    int lo = x, hi = x;
    for (int k = 1; k <= radius; ++k) {
      lo = lo == 0 ? n - 1 : lo - 1;
      hi = hi + 1 == n ? 0 : hi + 1;
      v += w[k] * (m[lo] + m[hi]);
    }
    out((size_t(z) * n + y) * n + x, v);
  }
}

__host__ __device__ inline size_t s1_smem(int n, int radius) {
  const size_t rows = size_t(kS1Rows + 2 * radius) * n + size_t(kS1Rows) * n, cols = size_t(32) * n;
  return (size_t(radius) + 1 + (rows > cols ? rows : cols)) * sizeof(double);
}

__global__ void __launch_bounds__(kS1Threads) k_s1_oc(const OCArgs A) {
  extern __shared__ __align__(16) unsigned char raw[];
  __shared__ double red[32];
  const int n = A.n, tid = threadIdx.x, radius = A.count;
  double* w = reinterpret_cast<double*>(raw);  // w[k]: tap at distance k
  double* buf = w + radius + 1;
  const size_t N = size_t(n) * n * n;
  const int columns = (n * n + 31) / 32, tasks = n * ((n + kS1Rows - 1) / kS1Rows);
  for (int k = tid; k <= radius; k += kS1Threads) w[k] = A.weights[radius + k];
  unsigned target = 0;
  for (int t = blockIdx.x; t < columns; t += gridDim.x) {
    s1_columns(buf, w, radius, n, t,
               [&](size_t i) { return A.dp[i] * 3 * (1. - 1e-4) * (A.ph[i] * A.ph[i]) * A.energy[i]; },
               [](size_t, double v) { return v; }, A.f2);
    s1_columns(buf, w, radius, n, t, [&](size_t i) { return A.dp[i]; }, [](size_t, double v) { return v; }, A.f3);
  }
  if (!grid_barrier(A.bar, target)) return oc_gave_up(A.bounds);
  // ratio = max(g, 1e-30) / max(dv, 1e-30); the upper bound is 1e4 times its maximum
  double m = 0.0;
  for (int t = blockIdx.x; t < tasks; t += gridDim.x) {
    s1_rows(buf, w, radius, n, t, A.f2, [&](size_t i, double v) { A.f0[i] = v; });
    s1_rows(buf, w, radius, n, t, A.f3, [&](size_t i, double v) {
      const double r = fmax(A.f0[i], 1e-30) / fmax(v, 1e-30);
      A.f0[i] = r;
      m = fmax(m, r);
    });
  }
  grid_max(m, A.bounds + 6);
  if (!grid_barrier(A.bar, target)) return oc_gave_up(A.bounds);
  double lo = 0.0, hi = __ldcg(A.bounds + 6) * 1e4;
  for (int it = 0; it < 45; ++it) {
    const double mid = (lo + hi) * 0.5, lam = fmax(mid, 1e-30);
    for (int t = blockIdx.x; t < columns; t += gridDim.x)
      s1_columns(buf, w, radius, n, t,
                 [&](size_t i) { return make_double2(A.x[i], __ldcg(A.f0 + i)); },
                 [&](size_t i, double2 xr) {
                   const double x = xr.x;
                   const double a = fmax(0., x - A.move), b = fmin(1., x + A.move);
                   const double v = fmin(b, fmax(a, x * sqrt(xr.y / lam)));
                   A.xnew[i] = v;
                   return v;
                 },
                 A.f2);
    if (!grid_barrier(A.bar, target)) return oc_gave_up(A.bounds);
    double acc[1] = {0.0};
    for (int t = blockIdx.x; t < tasks; t += gridDim.x)
      s1_rows(buf, w, radius, n, t, A.f2, [&](size_t, double v) {
        double p, d, a;
        s1_phys(v, A.beta, p, d, a);
        acc[0] += p;
      });
    block_sum<1>(acc, red);
    if (tid == 0) A.partials[blockIdx.x] = acc[0];
    if (!grid_barrier(A.bar, target)) return oc_gave_up(A.bounds);
    if (sum_partials(A.partials) / double(N) > A.volume) lo = mid; else hi = mid;
  }
  m = 0.0;
  for (size_t i = size_t(blockIdx.x) * kS1Threads + tid; i < N; i += size_t(gridDim.x) * kS1Threads)
    m = fmax(m, fabs(__ldcg(A.xnew + i) - A.x[i]));
  grid_max(m, A.bounds + 4);
  if (blockIdx.x == 0 && tid == 0 && !*(volatile int*)&A.bar->dead) {
    A.bounds[0] = lo;
    A.bounds[1] = hi;
    A.bounds[2] = 1.0;
    A.bounds[3] = 45.0;
  }
}

}  // namespace pgj

using namespace pgj;

namespace {
constexpr int kOCBlocks = 296;
// dynamic shared memory that needs no limit set: 48 KB less the kernels' static arrays
constexpr size_t kSmemAlways = 48 * 1024 - 384;
static_assert(sizeof(ConeSmem) <= kSmemAlways, "the cone filter needs no limit set");
// shared memory of a Study I block up to which the one-launch update is used: two blocks per SM (n = 128 with
// its own Gaussian takes 49 KB)
constexpr size_t kS1SmemMax = 100 * 1024;
const dim3 kConeBlock(kConeX, kConeY);
// Blocks that filter a field, at most `most`: one per tile of the tiled form; tables too long for it take up to one per
// plane of a tile.
int cone_blocks(int n, int count, int most) {
  return std::min(cone_tiles(n, count > kConeTaps ? 1 : kConeZ), most);
}

// Blocks of `fn` that are resident together on the current device with `smem` bytes each, at most
// kOCBlocks; 0 on error. Sets the kernel's shared memory limit. Asked on each call: the limit goes with the
// device's CUDA context when that is replaced (cudaDeviceReset).
int resident_blocks(const void* fn, int threads, size_t smem) {
  int device = 0, per = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e == cudaSuccess && smem > kSmemAlways)
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kS1SmemMax));
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, threads, smem);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (e != cudaSuccess) return set_cuda_error(e), 0;
  return std::min(kOCBlocks, per * sms);
}

int launch_cone(int n, const int32_t* offsets, const double* weights, int count, const double* x, double* y,
                cudaStream_t s) {
  k_cone_filter<<<cone_blocks(n, count, 4 * kOCBlocks), kConeBlock, sizeof(ConeSmem), s>>>(n, offsets, weights, count, x, y);
  return check_launch();
}

// One cooperative launch of an OC kernel with at most `work` blocks.
int launch_oc(const void* fn, dim3 block, size_t smem, size_t work, OCArgs& A, cudaStream_t s) {
  const int fit = resident_blocks(fn, int(block.x * block.y), smem);
  if (fit < 1) return PGJ_ERR_LAUNCH;
  void* args[] = {&A};
  const cudaError_t e = cudaLaunchCooperativeKernel(fn, dim3(unsigned(std::min(size_t(fit), work))), block, args, smem, s);
  return e == cudaSuccess ? PGJ_OK : set_cuda_error(e);
}
// scratch layout for the OC chains: 4 fields of N doubles, then 8 doubles of bisection state (lo, hi,
// continue flag, steps, change, -, largest ratio, -), the grid barrier's record (or a ticket) and
// kOCBlocks partials.
struct OCScratch {
  double *f0, *f1, *f2, *f3, *bounds, *partials;
  int* ticket;
};
OCScratch oc_scratch(double* scratch, size_t N) {
  OCScratch s;
  s.f0 = scratch; s.f1 = scratch + N; s.f2 = scratch + 2 * N; s.f3 = scratch + 3 * N;
  s.bounds = scratch + 4 * N;
  s.ticket = reinterpret_cast<int*>(s.bounds + 8);
  s.partials = s.bounds + 16;
  return s;
}

// Steps and change of a finished update; PGJ_ERR_TIMEOUT when a grid barrier gave up.
int read_record(const OCScratch& w, int* steps, double* change, cudaStream_t s) {
  double host[9];
  cudaError_t e = cudaMemcpyAsync(host, w.bounds, sizeof(host), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return set_cuda_error(e);
  GridBar bar;
  std::memcpy(&bar, host + 8, sizeof(bar));
  if (steps) *steps = int(host[3]);
  if (change) *change = host[4];
  return bar.dead ? PGJ_ERR_TIMEOUT : PGJ_OK;
}
}  // namespace

namespace pgj {
// `record`: 16 device doubles; *expired: the barrier gave up and left its mark
int grid_wait_selftest(int limit_us, double* record, bool* expired, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(record, 0, 16 * sizeof(double), s);
  if (e != cudaSuccess) return set_cuda_error(e);
  const unsigned long long limit = std::min(1000ull * static_cast<unsigned long long>(limit_us), kGridWaitNs);
  k_grid_wait_selftest<<<1, 32, 0, s>>>(reinterpret_cast<GridBar*>(record + 8), record, limit);
  int st = check_launch();
  if (st) return st;
  OCScratch w = {};
  w.bounds = record;
  int steps = 0;
  double change = 0.0;
  st = read_record(w, &steps, &change, s);
  *expired = st == PGJ_ERR_TIMEOUT && steps == -1 && std::isnan(change);
  return st == PGJ_ERR_TIMEOUT ? PGJ_OK : st;
}
}  // namespace pgj

extern "C" {

int pgj_cone_filter(int n, const int32_t* offsets, const double* weights, int count, const double* x, double* y,
                    void* stream) {
  if (n < 2 || !offsets || !weights || count < 1 || !x || !y) return PGJ_ERR_ARGUMENT;
  return launch_cone(n, offsets, weights, count, x, y, static_cast<cudaStream_t>(stream));
}

int pgj_paper_project(int n, const double* t, const double* hs, double beta, double eta, double emin, double* ph,
                      double* dp, double* a, void* stream) {
  if (n < 2 || !t || !hs || !ph || !dp || !a) return PGJ_ERR_ARGUMENT;
  k_paper_project<<<kOCBlocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(size_t(n) * n * n, t, hs, beta, eta, emin,
                                                                            ph, dp, a);
  return check_launch();
}

// scratch: 4 N + 16 + kOCBlocks doubles (see pgj.h: "4 n^3 float64" plus a small tail; callers
// allocate 4 n^3 + 512 doubles).
int pgj_paper_oc(int n, const int32_t* offsets, const double* weights, int count, const double* x, const double* ph,
                 const double* dp, const double* hs, const double* energy, double volume, double beta, double eta,
                 double emin, double move, double exponent, double floor_, double* xnew, double* scratch, int* steps,
                 double* change, void* stream) {
  if (n < 2 || !offsets || !weights || count < 1 || !x || !ph || !dp || !hs || !energy || !xnew || !scratch)
    return PGJ_ERR_ARGUMENT;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t N = size_t(n) * n * n;
  OCScratch w = oc_scratch(scratch, N);
  // bounds and the grid barrier's record
  cudaError_t e = cudaMemsetAsync(w.bounds, 0, 16 * sizeof(double), s);
  if (e != cudaSuccess) return set_cuda_error(e);
  OCArgs A = {};
  A.n = n;
  A.offsets = offsets; A.weights = weights; A.count = count;
  A.x = x; A.ph = ph; A.dp = dp; A.hs = hs; A.energy = energy;
  A.volume = volume; A.beta = beta; A.eta = eta; A.emin = emin; A.move = move; A.exponent = exponent; A.floor_ = floor_;
  A.xnew = xnew;
  A.f0 = w.f0; A.f1 = w.f1; A.f2 = w.f2; A.f3 = w.f3;
  A.bounds = w.bounds; A.bar = reinterpret_cast<GridBar*>(w.ticket); A.partials = w.partials;
  const size_t work = std::max<size_t>(cone_blocks(n, count, kOCBlocks), (N + kConeX * kConeY - 1) / (kConeX * kConeY));
  const int st = launch_oc(reinterpret_cast<const void*>(&k_paper_oc), kConeBlock, sizeof(ConeSmem), work, A, s);
  if (st) return st;
  if (!steps && !change) return PGJ_OK;  // enqueue only: the record stays in scratch[4N + 3 .. 4N + 4]
  return read_record(w, steps, change, s);
}

int pgj_gaussian_filter(int n, const double* weights, int radius, const double* x, double* y, double* scratch,
                        void* stream) {
  if (n < 2 || !weights || radius < 0 || 2 * radius + 1 > 4 * n + 1 || !x || !y || !scratch) return PGJ_ERR_ARGUMENT;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  k_gauss_axis<<<kOCBlocks, 256, 0, s>>>(n, 0, weights, radius, x, scratch);
  k_gauss_axis<<<kOCBlocks, 256, 0, s>>>(n, 1, weights, radius, scratch, scratch + size_t(n) * n * n);
  k_gauss_axis<<<kOCBlocks, 256, 0, s>>>(n, 2, weights, radius, scratch + size_t(n) * n * n, y);
  return check_launch();
}

int pgj_study1_project(int n, const double* t, double beta, double* ph, double* dp, double* a, void* stream) {
  if (n < 2 || !t || !ph || !dp || !a) return PGJ_ERR_ARGUMENT;
  k_s1_project<<<kOCBlocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(size_t(n) * n * n, t, beta, ph, dp, a);
  return check_launch();
}

int pgj_study1_oc(int n, const double* weights, int radius, const double* x, const double* ph, const double* dp,
                  const double* energy, double beta, double volume, double move, double* xnew, double* scratch,
                  double* change, void* stream) {
  if (n < 2 || !weights || radius < 0 || 2 * radius + 1 > 4 * n + 1 || !x || !ph || !dp || !energy || !xnew || !scratch)
    return PGJ_ERR_ARGUMENT;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t N = size_t(n) * n * n;
  OCScratch w = oc_scratch(scratch, N);
  cudaError_t e = cudaMemsetAsync(w.bounds, 0, 16 * sizeof(double), s);
  if (e != cudaSuccess) return set_cuda_error(e);
  if (s1_smem(n, radius) <= kS1SmemMax) {
    OCArgs A = {};
    A.n = n; A.weights = weights; A.count = radius;
    A.x = x; A.ph = ph; A.dp = dp; A.energy = energy;
    A.volume = volume; A.beta = beta; A.move = move; A.xnew = xnew;
    A.f0 = w.f0; A.f2 = w.f2; A.f3 = w.f3;
    A.bounds = w.bounds; A.bar = reinterpret_cast<GridBar*>(w.ticket); A.partials = w.partials;
    const size_t work = std::max<size_t>((size_t(n) * n + 31) / 32, size_t(n) * ((n + kS1Rows - 1) / kS1Rows));
    const int st1 = launch_oc(reinterpret_cast<const void*>(&k_s1_oc), dim3(kS1Threads), s1_smem(n, radius), work, A, s);
    if (st1 || !change) return st1;
    return read_record(w, nullptr, change, s);
  }
  // wider Gaussians than shared memory holds: separate passes over the fields (f0 ratio, f1 dv, f2/f3
  // filter temporaries; the Gaussian's scratch is f2|f3)
  k_s1_sens_in<<<kOCBlocks, 256, 0, s>>>(N, ph, dp, energy, xnew);
  int st;
  if ((st = pgj_gaussian_filter(n, weights, radius, xnew, w.f0, w.f2, stream))) return st;
  if ((st = pgj_gaussian_filter(n, weights, radius, dp, w.f1, w.f2, stream))) return st;
  k_s1_ratio<<<1, 1024, 0, s>>>(N, w.f0, w.f1, w.bounds);
  for (int it = 0; it < 45; ++it) {
    k_s1_candidate<<<kOCBlocks, 256, 0, s>>>(N, x, w.f0, w.bounds, move, xnew);
    if ((st = pgj_gaussian_filter(n, weights, radius, xnew, w.f1, w.f2, stream))) return st;
    k_s1_volume<<<kOCBlocks, 256, 0, s>>>(N, w.f1, beta, volume, w.bounds, w.partials, w.ticket);
  }
  // the candidate of the last bisection is the returned design (study.py:91-100)
  k_absmax_diff<<<1, 1024, 0, s>>>(N, xnew, x, w.bounds + 4);
  if ((st = check_launch())) return st;
  if (!change) return PGJ_OK;  // enqueue only: the change stays in scratch[4N + 4]
  return read_record(w, nullptr, change, s);
}

}  // extern "C"
