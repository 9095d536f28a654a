// The three transform kernels of one PCG iteration on grids whose load does not live in a cluster
// (pgj_resident.cuh), and of the first direction and true-residual replacements everywhere:
//
//   k_planes_fwd : r -= alpha q, ||r||^2, sum r -> last block: masks, mean r; 2D DFT over (x, y) of s.r
//   k_planes_z   : DFT along z, - mean r . DFT(s), symbol, <v, G v> and mean(s.w) by Parseval, inverse
//                  along z -> last block: rz, beta, mean(s.w)
//   k_planes_inv : inverse 2D DFT, d += alpha p, p = (s.w - mean(s.w)) + beta p; the WHILE condition
//
// (recurrence of resident.py:119-131 of exp/asg_gpu_resident_20261103; the two means of the projection P
// are exact identities in Fourier space, DFT(s.(r - m)) = DFT(s.r) - m DFT(s) and
// sum_x s.w = sum_k W(k) conj(DFT(s)(k)).)
//
// A block of the x/y kernels owns one component of two neighbouring z planes, packed as the real and
// imaginary parts of one complex plane: the whole plane is transformed in place in four passes (two
// factors per line, pgj_dft.cuh) and the two half spectra come apart as they are stored, so there is no
// packing of rows and no pass for the split. The half spectrum is (component, z, m) with m = ky ns + kx:
// the z kernel reads CS columns m of every plane as one contiguous run. The correction d takes its step
// in the inverse kernel, which reads p anyway (LoadScalars::step marks a load whose step is pending).
// Vectors are held by component, (3, N) per load, and move two values at a time.
//
// Bounds: each kernel moves its operands once; the x/y kernels are limited by the loads in flight that
// their planes leave room for (registers and shared memory), the z kernel by the same and, in FP64, by
// the arithmetic of the line transforms. Measured against the kernels they replace in pgj_planes.cu.
#pragma once
#include "pgj_internal.h"
#include "pgj_dft.cuh"

namespace pgj {

// kPlaneApply: z = P s G s P r of a caller's node-major FP64 vectors, all loads, no recurrence state. The mean of r
// comes from a pass of its own and leaves before the transforms: a recurrence's residual has next to none, a caller's
// vector may have one of any size, and taking that out in Fourier space would leave its rounding in z.
enum PlaneMode { kPlaneUpdate = 0, kPlaneInit = 1, kPlaneSync = 2, kPlaneScale = 3, kPlaneApply = 4 };

struct PlaneArgs {
  int lpd, loads, cap, mode, flex, init, set_cond, forward_only;
  void* p;                // (L, 3, N) T directions
  const void* q;          // (L, 3, N) T K p
  void* r;                // (L, 3, N) T residual
  void* d;                // (L, 3, N) T correction
  const double* r64;      // FP64 true residual, node-major (sync; FP64 init); apply: the caller's vector
  double* z64;            // apply: the caller's result
  const void* sp;         // (designs, 3, N) T scale
  void* spec;             // (L, 3, n, n ns) complex T
  const void* shat;       // (designs, 3, n, n ns) complex T: DFT of the scale
  void* zprev;            // flexible beta: (L, 3, N) T z of the previous direction
  const void* sym;        // (6, n, n ns) T
  const void* tw;         // n complex T
  LoadScalars* scal;
  const LoadScalars* out; // sync: certificate records
  double* partials;
  double rel_delta2;
  cudaGraphConditionalHandle h;  // inverse: the WHILE loop; forward: the replacement branch
  int* counters;
};

template <int N_, typename T_> struct PlaneCfg {
  using T = T_;
  static constexpr int N = N_, NN = N * N, NS = N / 2 + 1, M = N * NS, PX = N + 1;
  static constexpr int RA = Line<N>::RA, RB = Line<N>::RB;
  static constexpr size_t plane = size_t(N) * PX * 2 * sizeof(T);
  static constexpr size_t o_red = (plane + N * 2 * sizeof(T) + 15) / 16 * 16;
  static constexpr size_t smem = o_red + 4 * 32 * 8;
  // Blocks per SM: as many as keep their planes within 140 KB, at least two if they fit at all. The rest of an SM's
  // 256 KB is the L1 that the vectors pass through: with three FP64 blocks at n = 64 (200 KB of planes) the forward
  // and inverse kernels took 66 and 51 us, with two 52 and 41; n = 60 50 and 42 / 43 and 35; FP32 n = 90 86 and 86 /
  // 76 and 66. Below, the third block pays: n = 48 21 and 14 against 27 and 17 with two. Threads: a butterfly holds up
  // to 16 complex values, 64 registers in FP32, 85 in FP64; from 64 lines on 512 threads take a pass in one or two
  // rounds (FP64 n = 80 109 against 119 us with 384), below 384 have more registers (n = 60 78 against 81 us, both).
  static constexpr int fit = int((227 * 1024) / (smem + 1024));
  static constexpr int most = sizeof(T) == 4 ? 4 : 3, room = int((140 * 1024) / smem);
  static constexpr int MINB = room >= most ? most : room >= 3 ? 3 : fit >= 2 ? 2 : 1;
  static constexpr int NT = N <= 24 ? 128 : MINB >= 3 ? 256 : sizeof(T) == 8 && MINB == 2 && N < 64 ? 384 : 512;
  static_assert(fit >= 1, "a plane pair fits");
  // z kernel
  static constexpr int CS = sizeof(T) == 4 ? 32 : 16;
  static constexpr int ZT = (RA * CS + 31) / 32 * 32;
  static constexpr size_t o_zred = (size_t(3) * N * CS * 2 * sizeof(T) + N * 2 * sizeof(T) + 15) / 16 * 16;
  static constexpr size_t zsmem = o_zred + 4 * 32 * 8;
  static constexpr int zfit = int((227 * 1024) / (zsmem + 1024));
  static constexpr int zregs = sizeof(T) == 4 ? 80 : 168;
  static constexpr int ZB = (zfit < 65536 / (ZT * zregs) ? zfit : 65536 / (ZT * zregs)) < 1
                                ? 1
                                : (zfit < 65536 / (ZT * zregs) ? zfit : 65536 / (ZT * zregs));
};

// one pass over all lines of the plane in place; A / B: which factor; X: lines along x (lanes along y,
// the odd pitch keeps them on distinct banks) or along y (lanes along x)
template <class Cfg, bool INV, bool PASS_A, bool X>
__device__ __forceinline__ void plane_pass(cplx<typename Cfg::T>* buf, const cplx<typename Cfg::T>* tw) {
  using T = typename Cfg::T;
  using C = cplx<T>;
  constexpr int N = Cfg::N, RA = Cfg::RA, RB = Cfg::RB, PX = Cfg::PX;
  constexpr int R = PASS_A ? RA : RB, G = PASS_A ? RB : RA;  // points of a butterfly, butterflies of a line
  constexpr int step = PASS_A ? RB : 1, es = X ? 1 : PX, ls = X ? PX : 1;
  for (int w = threadIdx.x; w < G * N; w += Cfg::NT) {
    const int g = w / N, l = w - g * N;
    C* at = buf + l * ls + (PASS_A ? g : RB * g) * es;
    C v[R];
#pragma unroll
    for (int k = 0; k < R; ++k) v[k] = at[k * step * es];
    if constexpr (PASS_A) {
      if constexpr (INV) line_a_inv<T, N>(v, g, tw);
      else line_a<T, N>(v, g, tw);
    } else {
      Dft<T, R, INV>::run(v);
    }
#pragma unroll
    for (int k = 0; k < R; ++k) at[k * step * es] = v[k];
  }
}

template <class Cfg>
__global__ void __launch_bounds__(Cfg::NT, Cfg::MINB) k_planes_fwd(const __grid_constant__ PlaneArgs A) {
  using T = typename Cfg::T;
  using C = cplx<T>;
  constexpr int N = Cfg::N, NN = Cfg::NN, NT = Cfg::NT, NS = Cfg::NS, M = Cfg::M, PX = Cfg::PX;
  constexpr size_t NV = size_t(NN) * N, N3 = 3 * NV;
  constexpr int UNR = sizeof(T) == 4 ? 2 : 1;  // value pairs whose loads are in flight together
  extern __shared__ __align__(16) unsigned char smem[];
  const int c = blockIdx.x, z = 2 * blockIdx.y, load = blockIdx.z, tid = threadIdx.x;
  const int mode = A.mode;
  LoadScalars& S = A.scal[load];
  if (mode == kPlaneSync && A.set_cond && c == 0 && z == 0 && load == 0 && tid == 0) {
    A.counters[3] += 1;  // replacements taken (launch accounting)
    cudaGraphSetConditional(A.h, 0u);
  }
  if (mode == kPlaneSync ? S.reliable == 0 : (mode != kPlaneScale && mode != kPlaneApply && S.active == 0)) return;
  C* buf = reinterpret_cast<C*>(smem);
  C* tw = reinterpret_cast<C*>(smem + Cfg::plane);
  double* red = reinterpret_cast<double*>(smem + Cfg::o_red);
  for (int i = tid; i < N; i += NT) tw[i] = static_cast<const C*>(A.tw)[i];
  const size_t off = size_t(load) * N3 + size_t(c) * NV + size_t(z) * NN;  // plane a; plane b follows
  const size_t dsg = mode == kPlaneScale ? size_t(load) : size_t(load / A.lpd);
  const C* s2 = reinterpret_cast<const C*>(static_cast<const T*>(A.sp) + dsg * N3 + size_t(c) * NV + size_t(z) * NN);
  C* r2 = reinterpret_cast<C*>(static_cast<T*>(A.r) + off);
  double acc[3] = {0.0, 0.0, 0.0};
  constexpr int H = NN / 2;  // value pairs of a plane
  if (mode == kPlaneUpdate) {
    const C* q2 = reinterpret_cast<const C*>(static_cast<const T*>(A.q) + off);
    const T al = T(S.alpha);
    const C* zp = A.flex ? reinterpret_cast<const C*>(static_cast<const T*>(A.zprev) + off) : nullptr;
#pragma unroll 1
    for (int e0 = tid; e0 < H; e0 += UNR * NT) {
      C ra[UNR], rb[UNR], qa[UNR], qv[UNR], sa[UNR], sb[UNR];
#pragma unroll
      for (int u = 0; u < UNR; ++u) {
        const int e = e0 + u * NT;
        if (e >= H) continue;
        ra[u] = r2[e]; rb[u] = r2[H + e];
        qa[u] = q2[e]; qv[u] = q2[H + e];
        sa[u] = __ldg(s2 + e); sb[u] = __ldg(s2 + H + e);
      }
#pragma unroll
      for (int u = 0; u < UNR; ++u) {
        const int e = e0 + u * NT, y = e / (N / 2), x = 2 * (e - y * (N / 2));
        if (e >= H) continue;
        C a, b;
        a.x = ra[u].x - al * qa[u].x; a.y = ra[u].y - al * qa[u].y;
        b.x = rb[u].x - al * qv[u].x; b.y = rb[u].y - al * qv[u].y;
        r2[e] = a;
        r2[H + e] = b;
        const double ax = a.x, ay = a.y, bx = b.x, by = b.y;
        acc[0] += ax * ax + ay * ay + bx * bx + by * by;
        acc[1] += (ax + ay) + (bx + by);
        if (zp) {
          const C za = zp[e], zb = zp[H + e];
          acc[2] += ax * double(za.x) + ay * double(za.y) + bx * double(zb.x) + by * double(zb.y);
        }
        C* o = buf + y * PX + x;
        o[0] = cmk<C>(sa[u].x * a.x, sb[u].x * b.x);
        o[1] = cmk<C>(sa[u].y * a.y, sb[u].y * b.y);
      }
    }
  } else {
    // transform r as it stands: from the FP64 residual (sync; first direction in FP64), held (first
    // direction in FP32), or the scale itself
    const bool apply = sizeof(T) == 8 && mode == kPlaneApply;
    const bool from64 = mode == kPlaneSync || apply || (sizeof(T) == 8 && mode == kPlaneInit);
    const double* g = A.r64 + size_t(load) * N3 + 3 * (size_t(z) * NN) + c;
    const T m = apply ? T(S.mean_r[c]) : T(0);
#pragma unroll 2
    for (int e = tid; e < H; e += NT) {
      const int y = e / (N / 2), x = 2 * (e - y * (N / 2));
      const C sa = __ldg(s2 + e), sb = __ldg(s2 + H + e);
      C a = cmk<C>(T(1), T(1)), b = a;
      if (from64) {
        const double* ga = g + 6 * size_t(e);
        const double* gb = ga + 3 * size_t(NN);
        a = cmk<C>(T(ga[0]), T(ga[3]));
        b = cmk<C>(T(gb[0]), T(gb[3]));
        if (apply) {
          a = cmk<C>(a.x - m, a.y - m);
          b = cmk<C>(b.x - m, b.y - m);
        } else {
          r2[e] = a;
          r2[H + e] = b;
        }
      } else if (mode == kPlaneInit) {
        a = r2[e];
        b = r2[H + e];
      }
      C* o = buf + y * PX + x;
      o[0] = cmk<C>(sa.x * a.x, sb.x * b.x);
      o[1] = cmk<C>(sa.y * a.y, sb.y * b.y);
    }
  }
  __syncthreads();
  plane_pass<Cfg, false, true, true>(buf, tw);
  __syncthreads();
  plane_pass<Cfg, false, false, true>(buf, tw);
  __syncthreads();
  plane_pass<Cfg, false, true, false>(buf, tw);
  __syncthreads();
  plane_pass<Cfg, false, false, false>(buf, tw);
  __syncthreads();
  // A = (Z(k) + conj Z(-k)) / 2, B = (Z(k) - conj Z(-k)) / 2i
  C* sp = static_cast<C*>(A.spec) + ((size_t(load) * 3 + c) * N + z) * M;
#pragma unroll 2
  for (int k = tid; k < M; k += NT) {
    const int ky = k / NS, kx = k - ky * NS;
    const C zk = buf[line_pos<N>(ky) * PX + line_pos<N>(kx)];
    const C zn = buf[line_pos<N>(ky == 0 ? 0 : N - ky) * PX + line_pos<N>(kx == 0 ? 0 : N - kx)];
    sp[k] = cmk<C>(T(0.5) * (zk.x + zn.x), T(0.5) * (zk.y - zn.y));
    sp[M + k] = cmk<C>(T(0.5) * (zk.y + zn.y), T(0.5) * (zn.x - zk.x));
  }
  if (mode == kPlaneInit || mode == kPlaneScale || mode == kPlaneApply) return;

  const int nblk = 3 * (N / 2), blk = c + 3 * blockIdx.y;
  double* part = A.partials + size_t(load) * kPartialQ * kMaxPartials;
  if (mode == kPlaneUpdate) {
    block_sum<3>(acc, red);
    if (tid == 0) {
      part[blk] = acc[0];
      for (int cc = 0; cc < 3; ++cc) part[(1 + cc) * kMaxPartials + blk] = cc == c ? acc[1] : 0.0;
      part[4 * kMaxPartials + blk] = acc[2];
    }
    if (!last_block(&S.ticket[kTicketUpdate], nblk)) return;
    if (tid < 32) {
      double v[5];
#pragma unroll
      for (int k = 0; k < 5; ++k) v[k] = warp_sum_partials(part + k * kMaxPartials, nblk);
      if (tid == 0) {
        S.rz_cross = v[4];
        // same bookkeeping as the step-by-step update (k_update_ur)
        const double res2 = v[0];
        const bool finite = isfinite(res2);
        const int it = S.iterations + 1;
        const bool valid = S.failed == 0;
        const bool keep = valid && finite && (res2 > S.target2) && (it < A.cap);
        S.iterations = it;
        S.bad = S.bad | (valid ? 0 : 1) | (finite ? 0 : 1);
        S.active = keep ? 1 : 0;
        S.step = 1;
        S.res2 = res2;
        for (int cc = 0; cc < 3; ++cc) S.mean_r[cc] = v[1 + cc] / double(NV);
        if (A.rel_delta2 > 0.0) {
          const bool ok = valid && finite && it < A.cap;
          S.reliable = ok && ((keep && res2 < A.rel_delta2 * S.anchor) || (!keep && res2 <= S.target2)) ? 1 : 0;
          if (A.set_cond && S.reliable) cudaGraphSetConditional(A.h, 1u);  // some load takes a replacement
        }
      }
    }
  } else {  // the recurrence restarts from the FP64 true residual (as k_rel_sync)
    if (!last_block(&S.ticket[kTicketAux2], nblk)) return;
    if (tid == 0) {
      const LoadScalars& O = A.out[load];
      S.res2 = O.res2;
      S.anchor = O.res2;
      for (int cc = 0; cc < 3; ++cc) S.mean_r[cc] = O.mean_r[cc];
      S.active = isfinite(O.res2) && O.res2 > S.target2 && S.iterations < A.cap && !S.bad ? 1 : 0;
      S.reliable = 0;
      S.step = 0;  // the pending step went into the FP64 iterate with d
    }
  }
}

template <class Cfg>
__global__ void __launch_bounds__(Cfg::ZT, Cfg::ZB) k_planes_z(const __grid_constant__ PlaneArgs A) {
  using T = typename Cfg::T;
  using C = cplx<T>;
  constexpr int N = Cfg::N, ZT = Cfg::ZT, NS = Cfg::NS, M = Cfg::M, CS = Cfg::CS, RA = Cfg::RA, RB = Cfg::RB;
  extern __shared__ __align__(16) unsigned char smem[];
  const int load = blockIdx.y, tid = threadIdx.x;
  if (!A.forward_only && A.mode != kPlaneApply && A.scal[load].active == 0) return;
  C* buf = reinterpret_cast<C*>(smem);  // [component][z position][column]
  C* tw = buf + 3 * N * CS;
  double* red = reinterpret_cast<double*>(smem + Cfg::o_zred);
  for (int i = tid; i < N; i += ZT) tw[i] = static_cast<const C*>(A.tw)[i];
  const int m0 = blockIdx.x * CS, cnt = min(CS, M - m0);
  C* sp = static_cast<C*>(A.spec) + size_t(load) * 3 * N * M + m0;
  __syncthreads();
#pragma unroll 1
  for (int w = tid; w < 3 * RB * CS; w += ZT) {
    const int ml = w % CS, t = w / CS, b = t % RB, c = t / RB;
    if (ml >= cnt) continue;
    const C* src = sp + (size_t(c) * N + b) * M + ml;
    C v[RA];
#pragma unroll
    for (int k = 0; k < RA; ++k) v[k] = src[size_t(RB * k) * M];
    line_a<T, N>(v, b, tw);
    C* dst = buf + (c * N + b) * CS + ml;
#pragma unroll
    for (int k = 0; k < RA; ++k) dst[RB * k * CS] = v[k];
  }
  __syncthreads();
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  const C* sh = static_cast<const C*>(A.shat) + size_t(load / A.lpd) * 3 * N * M + m0;
  const T* sym = static_cast<const T*>(A.sym) + m0;
#pragma unroll 1
  for (int w = tid; w < RA * CS; w += ZT) {
    const int ml = w % CS, ka = w / CS;
    if (ml >= cnt) continue;
    C* at = buf + RB * ka * CS + ml;
    C v[3][RB];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
#pragma unroll
      for (int k = 0; k < RB; ++k) v[c][k] = at[(c * N + k) * CS];
      Dft<T, RB, false>::run(v[c]);
    }
    if (A.forward_only) {  // in place, wavenumbers in order
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int k = 0; k < RB; ++k) sp[(size_t(c) * N + ka + RA * k) * M + ml] = v[c][k];
      continue;
    }
    const int kx = (m0 + ml) % NS;
    const double wgt = (kx == 0 || kx == N / 2) ? 1.0 : 2.0;
    // DFT(s.(r - mean r)) = DFT(s.r) - mean r . DFT(s); apply: the mean is already out
    const bool out = A.mode == kPlaneApply;
    const T mx = out ? T(0) : T(A.scal[load].mean_r[0]), my = out ? T(0) : T(A.scal[load].mean_r[1]);
    const T mz = out ? T(0) : T(A.scal[load].mean_r[2]);
    double part[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int k = 0; k < RB; ++k) {
      const size_t kk = size_t(ka + RA * k) * M + ml;
      constexpr size_t Nh = size_t(N) * M;
      const T c0 = __ldg(sym + kk), c1 = __ldg(sym + Nh + kk), c2 = __ldg(sym + 2 * Nh + kk);
      const T c3 = __ldg(sym + 3 * Nh + kk), c4 = __ldg(sym + 4 * Nh + kk), c5 = __ldg(sym + 5 * Nh + kk);
      const C s0 = __ldg(sh + kk), s1 = __ldg(sh + Nh + kk), s2 = __ldg(sh + 2 * Nh + kk);
      const C x = cmk<C>(v[0][k].x - mx * s0.x, v[0][k].y - mx * s0.y);
      const C y = cmk<C>(v[1][k].x - my * s1.x, v[1][k].y - my * s1.y);
      const C z = cmk<C>(v[2][k].x - mz * s2.x, v[2][k].y - mz * s2.y);
      const C wx = cmk<C>(c0 * x.x + c3 * y.x + c4 * z.x, c0 * x.y + c3 * y.y + c4 * z.y);
      const C wy = cmk<C>(c3 * x.x + c1 * y.x + c5 * z.x, c3 * x.y + c1 * y.y + c5 * z.y);
      const C wz = cmk<C>(c4 * x.x + c5 * y.x + c2 * z.x, c4 * x.y + c5 * y.y + c2 * z.y);
      part[0] += double(x.x) * wx.x + double(x.y) * wx.y + double(y.x) * wy.x + double(y.y) * wy.y +
                 double(z.x) * wz.x + double(z.y) * wz.y;
      // sum_x s w = sum_k W conj(DFT(s)) (1/N is folded into the symbol)
      part[1] += double(wx.x) * s0.x + double(wx.y) * s0.y;
      part[2] += double(wy.x) * s1.x + double(wy.y) * s1.y;
      part[3] += double(wz.x) * s2.x + double(wz.y) * s2.y;
      v[0][k] = wx; v[1][k] = wy; v[2][k] = wz;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) acc[k] += wgt * part[k];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      Dft<T, RB, true>::run(v[c]);
#pragma unroll
      for (int k = 0; k < RB; ++k) at[(c * N + k) * CS] = v[c][k];
    }
  }
  if (A.forward_only) return;
  __syncthreads();
#pragma unroll 1
  for (int w = tid; w < 3 * RB * CS; w += ZT) {
    const int ml = w % CS, t = w / CS, b = t % RB, c = t / RB;
    if (ml >= cnt) continue;
    const C* src = buf + (c * N + b) * CS + ml;
    C v[RA];
#pragma unroll
    for (int k = 0; k < RA; ++k) v[k] = src[RB * k * CS];
    line_a_inv<T, N>(v, b, tw);
    C* dst = sp + (size_t(c) * N + b) * M + ml;
#pragma unroll
    for (int k = 0; k < RA; ++k) dst[size_t(RB * k) * M] = v[k];
  }
  // Parseval partials -> last block: rz, beta, mean(s.w)
  block_sum<4>(acc, red);
  const int nblk = gridDim.x, blk = blockIdx.x;
  double* part = A.partials + size_t(load) * kPartialQ * kMaxPartials;
  if (tid == 0)
    for (int k = 0; k < 4; ++k) part[k * kMaxPartials + blk] = acc[k];
  LoadScalars& S = A.scal[load];
  if (!last_block(&S.ticket[kTicketFZ], nblk)) return;
  if (tid < 32) {
    double v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = warp_sum_partials(part + k * kMaxPartials, nblk);
    if (tid == 0) {
      if (A.mode == kPlaneApply) {
      } else if (A.init) {
        S.beta = 0.0;
      } else {
        const double rz = S.rz;
        S.beta = (A.flex ? v[0] - S.rz_cross : v[0]) / (rz != 0.0 ? rz : 1.0);
      }
      if (A.mode != kPlaneApply) S.rz = v[0];
      for (int k = 0; k < 3; ++k) S.mean_z[k] = v[1 + k] / double(size_t(N) * N * N);
    }
  }
}

template <class Cfg>
__global__ void __launch_bounds__(Cfg::NT, Cfg::MINB) k_planes_inv(const __grid_constant__ PlaneArgs A) {
  using T = typename Cfg::T;
  using C = cplx<T>;
  constexpr int N = Cfg::N, NN = Cfg::NN, NT = Cfg::NT, NS = Cfg::NS, M = Cfg::M, PX = Cfg::PX;
  constexpr size_t NV = size_t(NN) * N, N3 = 3 * NV;
  constexpr int H = NN / 2;
  extern __shared__ __align__(16) unsigned char smem[];
  const int c = blockIdx.x, z = 2 * blockIdx.y, load = blockIdx.z, tid = threadIdx.x;
  if (A.set_cond && c == 0 && z == 0 && load == 0 && tid == 0) {
    int any = 0;
    for (int l = 0; l < A.loads; ++l) any |= A.scal[l].active;
    if (A.init) {
      cudaGraphSetConditional(A.h, any ? 1u : 0u);  // the attempt's loop, which the last attempt left at 0
    } else {
      const int runs = ++A.counters[0];
      A.counters[5] += 1;                          // loop bodies over the whole solve
      if (runs >= A.cap + 100) A.counters[1] = 1;  // recorded: loop stopped by the bound
      cudaGraphSetConditional(A.h, (any && runs < A.cap + 100) ? 1u : 0u);
    }
  }
  const LoadScalars& S = A.scal[load];
  const bool apply = sizeof(T) == 8 && A.mode == kPlaneApply;
  const bool step = !apply && S.step != 0, active = apply || S.active != 0;
  if (!step && !active) return;
  const size_t off = size_t(load) * N3 + size_t(c) * NV + size_t(z) * NN;
  C* d2 = reinterpret_cast<C*>(static_cast<T*>(A.d) + off);
  C* p2 = reinterpret_cast<C*>(static_cast<T*>(A.p) + off);
  const T al = T(S.alpha);
  if (!active) {  // the load stopped with this step
    for (int e = tid; e < H; e += NT) {
      const C da = d2[e], db = d2[H + e], pa = p2[e], pb = p2[H + e];
      d2[e] = cmk<C>(da.x + al * pa.x, da.y + al * pa.y);
      d2[H + e] = cmk<C>(db.x + al * pb.x, db.y + al * pb.y);
    }
    return;
  }
  C* buf = reinterpret_cast<C*>(smem);
  C* tw = reinterpret_cast<C*>(smem + Cfg::plane);
  for (int i = tid; i < N; i += NT) tw[i] = static_cast<const C*>(A.tw)[i];
  const C* sp = static_cast<const C*>(A.spec) + ((size_t(load) * 3 + c) * N + z) * M;
  // Z = A + i B over the whole plane from the two half spectra
  constexpr int UF = sizeof(T) == 8 ? 2 : 4;  // points whose loads are in flight together
#pragma unroll 1
  for (int w0 = tid; w0 < M; w0 += UF * NT) {
    C va[UF], vb[UF];
#pragma unroll
    for (int u = 0; u < UF; ++u) {
      const int k = w0 + u * NT;
      if (k < M) { va[u] = sp[k]; vb[u] = sp[M + k]; }
    }
#pragma unroll
    for (int u = 0; u < UF; ++u) {
      const int k = w0 + u * NT, ky = k / NS, kx = k - ky * NS;
      if (k >= M) continue;
      buf[line_pos<N>(ky) * PX + line_pos<N>(kx)] = cmk<C>(va[u].x - vb[u].y, va[u].y + vb[u].x);
      if (kx != 0 && kx != N / 2)
        buf[line_pos<N>(ky == 0 ? 0 : N - ky) * PX + line_pos<N>(N - kx)] =
            cmk<C>(va[u].x + vb[u].y, vb[u].x - va[u].y);
    }
  }
  __syncthreads();
  plane_pass<Cfg, true, false, false>(buf, tw);
  __syncthreads();
  plane_pass<Cfg, true, true, false>(buf, tw);
  __syncthreads();
  plane_pass<Cfg, true, false, true>(buf, tw);
  __syncthreads();
  plane_pass<Cfg, true, true, true>(buf, tw);
  __syncthreads();
  const C* s2 = reinterpret_cast<const C*>(static_cast<const T*>(A.sp) + size_t(load / A.lpd) * N3 + size_t(c) * NV + size_t(z) * NN);
  C* zp = A.flex ? reinterpret_cast<C*>(static_cast<T*>(A.zprev) + off) : nullptr;
  const T m = T(S.mean_z[c]), beta = T(S.beta);
  const bool init = A.init != 0;
  constexpr int UNR = sizeof(T) == 4 ? 2 : 1;
#pragma unroll 1
  for (int e0 = tid; e0 < H; e0 += UNR * NT) {
    C sa[UNR], sb[UNR], da[UNR], db[UNR], pa[UNR], pb[UNR];
#pragma unroll
    for (int u = 0; u < UNR; ++u) {
      const int e = e0 + u * NT;
      if (e >= H) continue;
      sa[u] = __ldg(s2 + e); sb[u] = __ldg(s2 + H + e);
      pa[u] = pb[u] = cmk<C>(T(0), T(0));
      if (!init) { pa[u] = p2[e]; pb[u] = p2[H + e]; }
      if (step) { da[u] = d2[e]; db[u] = d2[H + e]; }
    }
#pragma unroll
    for (int u = 0; u < UNR; ++u) {
      const int e = e0 + u * NT, y = e / (N / 2), x = 2 * (e - y * (N / 2));
      if (e >= H) continue;
      if (step) {
        d2[e] = cmk<C>(da[u].x + al * pa[u].x, da[u].y + al * pa[u].y);
        d2[H + e] = cmk<C>(db[u].x + al * pb[u].x, db[u].y + al * pb[u].y);
      }
      const C w0 = buf[y * PX + x], w1 = buf[y * PX + x + 1];
      const C za = cmk<C>(sa[u].x * w0.x - m, sa[u].y * w1.x - m), zb = cmk<C>(sb[u].x * w0.y - m, sb[u].y * w1.y - m);
      if (apply) {
        double* o = A.z64 + size_t(load) * N3 + 3 * (size_t(z) * NN) + c + 6 * size_t(e);
        o[0] = za.x; o[3] = za.y;
        o[3 * size_t(NN)] = zb.x; o[3 * size_t(NN) + 3] = zb.y;
        continue;
      }
      p2[e] = cmk<C>(za.x + beta * pa[u].x, za.y + beta * pa[u].y);
      p2[H + e] = cmk<C>(zb.x + beta * pb[u].x, zb.y + beta * pb[u].y);
      if (zp) {
        zp[e] = za;
        zp[H + e] = zb;
      }
    }
  }
}

// The kernels of a grid and precision, with their launch shapes.
struct PlaneKernels {
  const void *fwd, *z, *inv;
  int n, prec, nt, zt, cs, m;
  size_t smem, zsmem;
};

template <class Cfg> PlaneKernels planes_entry() {
  PlaneKernels k;
  k.fwd = reinterpret_cast<const void*>(&k_planes_fwd<Cfg>);
  k.z = reinterpret_cast<const void*>(&k_planes_z<Cfg>);
  k.inv = reinterpret_cast<const void*>(&k_planes_inv<Cfg>);
  k.n = Cfg::N;
  k.prec = sizeof(typename Cfg::T) == 4 ? PGJ_FP32 : PGJ_FP64;
  k.nt = Cfg::NT;
  k.zt = Cfg::ZT;
  k.cs = Cfg::CS;
  k.m = Cfg::M;
  k.smem = Cfg::smem;
  k.zsmem = Cfg::zsmem;
  return k;
}

}  // namespace pgj
