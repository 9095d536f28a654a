// Matrix-free periodic HEX8 operator q = K(a) p, two elements of a row per thread.
//
// A block owns TY node rows of full length n and marches a chunk of z planes: (TY + 1) x n / 2 threads, the
// first row of threads being the element row below the tile (a halo, its upper forces only). A thread
// owns the elements (x, x + 1) of one element row, x even, and reads the three nodes of each of its two
// node rows straight from global memory: pairs are 8- or 16-byte aligned for every even n, neighbours hit
// the L1, and the values of the next plane are in flight while this one is computed. Both elements go
// through the modal action (element_modal) as one packed pair: in FP32 every add, multiply and fused
// multiply-add is one instruction for both.
//
// The lower and upper face modes of a column stay in registers from plane to plane. Per plane the forces on
// the lower face are summed along x inside the thread, and what belongs to other threads goes through
// shared memory, double-buffered over one barrier: the forces on the right neighbour's node, those on the
// node row above, and the corner of both. Fixed summation order, no atomics (unlike the scatter of
// exp/asg_gpu_resident_20261103/scalar_fi.cu:14-36).
//
// One element per thread with the node planes staged in shared memory spent its time on the exchange (9
// values an element, now 4.5) and on shared loads. Recurrence operator of six loads, us, that form / this one:
// FP64 n = 48 31 / 22.7, 64 59 / 45, 72 92 / 57, 96 172 / 131; FP32 n = 48 26.5 / 16.5, 64 37 / 26.8, 72 74 / 36,
// 96 133 / 88, 128 294 / 205. Eight (FP64) or twelve warps per SM at 150 to 250 registers bound it: the serial
// chain of a plane step (loads, modal action, exchange, barrier) is covered by few others. Leaving the halo
// row out and having the update kernel add the missing rows of q was no faster over both kernels (n = 64 FP64
// 109 against 112 us, FP32 53 against 54; n = 96 338 against 317, 199 against 179).
#pragma once
#include "pgj_internal.h"

namespace pgj {

// Values of the two elements (or nodes) of a thread.
template <typename R> struct Pair;
template <> struct Pair<float> {
  float2 v;
  static __device__ __forceinline__ Pair make(float a, float b) { return Pair{make_float2(a, b)}; }
  static __device__ __forceinline__ Pair all(float a) { return make(a, a); }
  __device__ __forceinline__ float a() const { return v.x; }
  __device__ __forceinline__ float b() const { return v.y; }
  friend __device__ __forceinline__ Pair operator+(Pair p, Pair q) { return Pair{__fadd2_rn(p.v, q.v)}; }
  friend __device__ __forceinline__ Pair operator-(Pair p, Pair q) {
    return Pair{__ffma2_rn(q.v, make_float2(-1.f, -1.f), p.v)};  // one instruction, rounds like a subtraction
  }
  friend __device__ __forceinline__ Pair operator*(Pair p, Pair q) { return Pair{__fmul2_rn(p.v, q.v)}; }
  static __device__ __forceinline__ Pair fma(Pair p, Pair q, Pair r) { return Pair{__ffma2_rn(p.v, q.v, r.v)}; }
};
template <> struct Pair<double> {
  double x, y;
  static __device__ __forceinline__ Pair make(double a, double b) { return Pair{a, b}; }
  static __device__ __forceinline__ Pair all(double a) { return make(a, a); }
  __device__ __forceinline__ double a() const { return x; }
  __device__ __forceinline__ double b() const { return y; }
  friend __device__ __forceinline__ Pair operator+(Pair p, Pair q) { return Pair{p.x + q.x, p.y + q.y}; }
  friend __device__ __forceinline__ Pair operator-(Pair p, Pair q) { return Pair{p.x - q.x, p.y - q.y}; }
  friend __device__ __forceinline__ Pair operator*(Pair p, Pair q) { return Pair{p.x * q.x, p.y * q.y}; }
  static __device__ __forceinline__ Pair fma(Pair p, Pair q, Pair r) {
    return Pair{::fma(p.x, q.x, r.x), ::fma(p.y, q.y, r.y)};
  }
};

// element_modal (pgj_common.cuh) of two elements at once
template <typename R>
__device__ __forceinline__ void element_modal2(const Pair<R> (&Q)[8][3], Pair<R> A, const OpConst& k, Pair<R> (&P)[8][3]) {
  using V = Pair<R>;
  const V l0 = A * V::all(R(k.l0)), m0 = A * V::all(R(k.m0)), m20 = m0 + m0;
  const V lt = l0 * (Q[1][0] + Q[2][1] + Q[4][2]);
  const V gyz = m0 * (Q[4][1] + Q[2][2]), gxz = m0 * (Q[4][0] + Q[1][2]), gxy = m0 * (Q[2][0] + Q[1][1]);
  P[1][0] = V::fma(m20, Q[1][0], lt); P[1][1] = gxy; P[1][2] = gxz;
  P[2][0] = gxy; P[2][1] = V::fma(m20, Q[2][1], lt); P[2][2] = gyz;
  P[4][0] = gxz; P[4][1] = gyz; P[4][2] = V::fma(m20, Q[4][2], lt);
  const V l1 = A * V::all(R(k.l1)), m1 = A * V::all(R(k.m1)), n1 = A * V::all(R(k.n1));
  P[3][0] = V::fma(n1, Q[3][0], l1 * Q[6][2]);
  P[3][1] = V::fma(n1, Q[3][1], l1 * Q[5][2]);
  P[5][0] = V::fma(n1, Q[5][0], l1 * Q[6][1]);
  P[5][2] = V::fma(n1, Q[5][2], l1 * Q[3][1]);
  P[6][1] = V::fma(n1, Q[6][1], l1 * Q[5][0]);
  P[6][2] = V::fma(n1, Q[6][2], l1 * Q[3][0]);
  const V S = Q[3][2] + Q[5][1] + Q[6][0];
  P[3][2] = m1 * (S + Q[3][2]);
  P[5][1] = m1 * (S + Q[5][1]);
  P[6][0] = m1 * (S + Q[6][0]);
  const V k7 = A * V::all(R(k.k7));
  P[7][0] = k7 * Q[7][0]; P[7][1] = k7 * Q[7][1]; P[7][2] = k7 * Q[7][2];
}

// The three nodes (x, x + 1, x + 2) of one row: a pair and the next value, per component.
template <typename T> struct RowNodes {
  T v[3][3];  // [component][node]
};
// IL: node-major (x, y, z interleaved); otherwise by component, `N` values each. VEC: pairs are aligned.
template <typename T, bool IL, bool VEC>
__device__ __forceinline__ RowNodes<T> load_row(const T* __restrict__ in, unsigned N, unsigned row, unsigned x0, unsigned x2) {
  using C = cplx<T>;
  RowNodes<T> r;
  if constexpr (!VEC) {
    static_assert(IL || VEC, "vectors by component are the library's own");
    const T* p = in + 3 * (row + x0);
    const T* e = in + 3 * (row + x2);
#pragma unroll
    for (int c = 0; c < 3; ++c) { r.v[c][0] = p[c]; r.v[c][1] = p[3 + c]; r.v[c][2] = e[c]; }
  } else if constexpr (IL) {
    const C* p = reinterpret_cast<const C*>(in + 3 * (row + x0));
    const C a = p[0], b = p[1], c = p[2];
    const T* e = in + 3 * (row + x2);
    r.v[0][0] = a.x; r.v[1][0] = a.y; r.v[2][0] = b.x;
    r.v[0][1] = b.y; r.v[1][1] = c.x; r.v[2][1] = c.y;
    r.v[0][2] = e[0]; r.v[1][2] = e[1]; r.v[2][2] = e[2];
  } else {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const C a = *reinterpret_cast<const C*>(in + c * N + row + x0);
      r.v[c][0] = a.x;
      r.v[c][1] = a.y;
      r.v[c][2] = in[c * N + row + x2];
    }
  }
  return r;
}

// T: storage of p and q, R: arithmetic (double with T = float for high-contrast mixed solves). COMP: p and q
// held by component, (3, N) per load; otherwise node-major. VEC: p and q are aligned to pairs (a caller's vectors
// need not be). THR: most threads of a block.
template <typename T, int MODE, typename R, bool COMP, bool VEC, int THR>
__global__ void __launch_bounds__(THR, 1) k_rows(const StencilArgs A) {
  using V = Pair<R>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n = A.n, TY = A.ty, nh = n >> 1;
  const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + nh * ty;
  const int load = blockIdx.z;
  const int nblk = gridDim.x * gridDim.y, blk = blockIdx.x + gridDim.x * blockIdx.y;
  const size_t N = size_t(n) * n * n;
  const int y0 = blockIdx.x * TY, z0 = blockIdx.y * A.zc;
  const int zc = min(A.zc, n - z0);
  const int ey = y0 - 1 + ty;  // element row = own node row
  const int eyw = ey < 0 ? n - 1 : (ey >= n ? ey % n : ey), eyp = eyw + 1 == n ? 0 : eyw + 1;
  const bool out_row = ty >= 1 && ey < n;
  const int x0 = 2 * tx, x2 = x0 + 2 == n ? 0 : x0 + 2;

  bool act = true;
  if (MODE == kPCG) act = A.scal[load].active != 0;
  else if (A.active_ext) act = A.active_ext[load] != 0;
  else if (MODE == kResidual && A.rel_flags) act = A.rel_flags[load].reliable != 0;
  // certification of a batched context: a design that took its last attempt keeps its certificate
  if (MODE == kResidual && A.scal[load].frozen) act = false;
  T* out = reinterpret_cast<T*>(A.out) + size_t(load) * 3 * N;
  if (!act) {
    if (MODE == kPCG && blk == 0 && tid == 0) A.scal[load].step = 0;  // its last step has been taken
    if (MODE == kPlain && out_row)
      for (int z = z0; z < z0 + zc; ++z) {
        T* o = out + 3 * ((size_t(z) * n + ey) * n + x0);
#pragma unroll
        for (int k = 0; k < 6; ++k) o[k] = T(0);
      }
    return;
  }
  const T* in = reinterpret_cast<const T*>(A.in) + size_t(load) * 3 * N;

  // exchange, double-buffered: [parity][12 values][THR threads], in the order up (3 pairs), right (3),
  // corner (3); the constant stride puts the offsets into the instructions
  R* xb = reinterpret_cast<R*>(smem_raw);
  R* xo = xb + 12 * THR;
  double* red = reinterpret_cast<double*>(xb + 24 * THR);
  const int left = tx == 0 ? nh - 1 : tx - 1;
  const int t_left = ty * nh + left, t_below = (ty >= 1 ? ty - 1 : 0) * nh;

  const double* arow = A.a + size_t(load / A.lpd) * N + size_t(eyw) * n + x0;
  // offsets within a load's vector stay below 3 * 256^3 and take 32 bits
  const unsigned plane = unsigned(n) * n, uN = unsigned(N);
  const unsigned r0 = unsigned(eyw) * n, r1 = unsigned(eyp) * n;
  // planes z0 - 1 (only its element plane's upper forces matter) .. z0 + zc
  unsigned z = z0 == 0 ? n - 1 : z0 - 1;
  RowNodes<T> na = load_row<T, !COMP, VEC>(in, uN, z * plane + r0, x0, x2), nb = load_row<T, !COMP, VEC>(in, uN, z * plane + r1, x0, x2);
  double2 an = __ldg(reinterpret_cast<const double2*>(arow + z * plane));
  V F0[4][3], Up[4][3], own[3];
  auto faces = [&](const RowNodes<T>& a, const RowNodes<T>& b, V (&F)[4][3]) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const V u0 = V::make(R(a.v[c][0]), R(a.v[c][1])), u1 = V::make(R(b.v[c][0]), R(b.v[c][1]));
      const R a2 = R(a.v[c][2]), b2 = R(b.v[c][2]);
      const V s = u1 + u0, d = u1 - u0;              // over y at x, x + 1
      const V ss = V::make(s.b(), b2 + a2), ds = V::make(d.b(), b2 - a2);  // at x + 1, x + 2
      F[0][c] = ss + s;
      F[1][c] = ss - s;
      F[2][c] = ds + d;
      F[3][c] = ds - d;
    }
  };
  faces(na, nb, F0);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    own[c] = V::all(R(0));
#pragma unroll
    for (int f = 0; f < 4; ++f) Up[f][c] = V::all(R(0));
  }
  z = z + 1 == unsigned(n) ? 0 : z + 1;
  na = load_row<T, !COMP, VEC>(in, uN, z * plane + r0, x0, x2);
  nb = load_row<T, !COMP, VEC>(in, uN, z * plane + r1, x0, x2);
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 1
  for (int s = 0; s <= zc; ++s) {
    // element plane z0 - 1 + s, upper node plane z (its rows are in na, nb)
    const V ae = V::make(R(an.x), R(an.y));
    V F1[4][3], own1[3];
    faces(na, nb, F1);
#pragma unroll
    for (int c = 0; c < 3; ++c) own1[c] = V::make(R(na.v[c][0]), R(na.v[c][1]));
    if (s < zc) {  // the next plane's values
      an = __ldg(reinterpret_cast<const double2*>(arow + z * plane));
      z = z + 1 == unsigned(n) ? 0 : z + 1;
      na = load_row<T, !COMP, VEC>(in, uN, z * plane + r0, x0, x2);
      nb = load_row<T, !COMP, VEC>(in, uN, z * plane + r1, x0, x2);
    }
    V Q[8][3], P[8][3];
#pragma unroll
    for (int f = 0; f < 4; ++f)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        Q[f][c] = F1[f][c] + F0[f][c];
        Q[f + 4][c] = F1[f][c] - F0[f][c];
        F0[f][c] = F1[f][c];
      }
    element_modal2<R>(Q, ae, A.kc, P);
    V low[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      V G[4];
      // P[0] = 0: the constant mode carries no strain
      G[0] = Up[0][c] - P[4][c];
      Up[0][c] = P[4][c];
#pragma unroll
      for (int f = 1; f < 4; ++f) {
        G[f] = (P[f][c] - P[f + 4][c]) + Up[f][c];
        Up[f][c] = P[f][c] + P[f + 4][c];
      }
      // lower face: corners (x, y), (x + 1, y), (x, y + 1), (x + 1, y + 1) of both elements
      const V l0 = G[0] - G[2], l1 = G[1] - G[3], u0 = G[0] + G[2], u1 = G[1] + G[3];
      const V c00 = l0 - l1, c10 = l0 + l1, c01 = u0 - u1, c11 = u0 + u1;
      low[c] = V::make(c00.a(), c00.b() + c10.a());
      if (s >= 1) {
        reinterpret_cast<V*>(xb)[c * THR + tid] = V::make(c01.a(), c01.b() + c11.a());
        xb[(6 + c) * THR + tid] = c10.b();
        xb[(9 + c) * THR + tid] = c11.b();
      }
    }
    __syncthreads();  // forces published; the other parity's are free again
    if (s >= 1 && out_row) {
      const unsigned node = (unsigned(z0 + s - 1) * n + ey) * n + x0;
      V q[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const V lu = low[c] + reinterpret_cast<const V*>(xb)[c * THR + t_below + tx];
        const R e = xb[(6 + c) * THR + t_left] + xb[(9 + c) * THR + t_below + left];
        q[c] = V::make(lu.a() + e, lu.b());
      }
      if (MODE == kResidual) {
        const double* fl = A.f + size_t(load) * 3 * N + 3 * node;
        T* o = out + 3 * node;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const double ra = fl[c] - double(q[c].a()), rb = fl[3 + c] - double(q[c].b());
          o[c] = T(ra);
          o[3 + c] = T(rb);
          acc[0] += ra * ra + rb * rb;
          acc[1 + c] += ra + rb;
        }
      } else {
        if constexpr (COMP) {
#pragma unroll
          for (int c = 0; c < 3; ++c)
            *reinterpret_cast<cplx<T>*>(out + (c * uN + node)) = cmk<cplx<T>>(T(q[c].a()), T(q[c].b()));
        } else if constexpr (!VEC) {
          T* o = out + 3 * node;
#pragma unroll
          for (int c = 0; c < 3; ++c) { o[c] = T(q[c].a()); o[3 + c] = T(q[c].b()); }
        } else {
          cplx<T>* o = reinterpret_cast<cplx<T>*>(out + 3 * node);
          o[0] = cmk<cplx<T>>(T(q[0].a()), T(q[1].a()));
          o[1] = cmk<cplx<T>>(T(q[2].a()), T(q[0].b()));
          o[2] = cmk<cplx<T>>(T(q[1].b()), T(q[2].b()));
        }
        if (MODE == kPCG)
#pragma unroll
          for (int c = 0; c < 3; ++c)
            acc[0] += double(own[c].a()) * double(q[c].a()) + double(own[c].b()) * double(q[c].b());
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) own[c] = own1[c];
    R* t = xb;
    xb = xo;
    xo = t;
  }

  if (MODE == kPlain) return;
  block_sum<4>(acc, red);
  double* part = A.partials + size_t(load) * kPartialQ * kMaxPartials;
  if (tid == 0) {
#pragma unroll
    for (int k = 0; k < 4; ++k) part[k * kMaxPartials + blk] = acc[k];
  }
  LoadScalars& S = A.scal[load];
  if (!last_block(&S.ticket[kTicketApply], nblk)) return;
  if (tid < 32) {
    if (MODE == kPCG) {
      const double den = warp_sum_partials(part, nblk);
      if (tid == 0) {
        const double rz = S.rz;
        const bool valid = isfinite(den) && den > 0.0 && isfinite(rz) && rz > 0.0;
        S.failed = valid ? 0 : 1;
        S.alpha = valid ? rz / den : 0.0;
      }
    } else {
      double v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] = warp_sum_partials(part + k * kMaxPartials, nblk);
      if (tid == 0) {
        S.res2 = v[0];
        S.absolute = sqrt(v[0]);
        const double inv = 1.0 / double(N);
#pragma unroll
        for (int c = 0; c < 3; ++c) S.mean_r[c] = v[1 + c] * inv;
      }
    }
  }
}

}  // namespace pgj
