// In-register DFTs of a fixed radix and the two-factor line transform built from them.
//
// A line of N = RA * RB points is transformed in place by two passes over memory, whatever holds it:
//   pass A, for each b < RB : DFT_RA over the points RB a + b, times W_N^(b ka), back to RB ka + b
//   pass B, for each ka < RA: DFT_RB over the points RB ka + b, back to RB ka + kb
// after which position RB ka + kb holds X[ka + RA kb]. The inverse runs the passes backwards on that
// order and leaves natural order. Every butterfly reads and writes the same positions, so a pass needs
// no second buffer, and the order of the spectrum only shows where it is read or stored (line_pos).
#pragma once
#include "pgj_common.cuh"

namespace pgj {

// v[k] <- sum_j v[j] e^(-+ 2 pi i jk / R) (INV: the conjugate, unnormalised)
template <typename T, int R, bool INV> struct Dft;

template <typename C, bool INV> __device__ __forceinline__ C rot90(C a) {  // times -i (forward) or +i
  return INV ? cmk<C>(-a.y, a.x) : cmk<C>(a.y, -a.x);
}

template <typename T, bool INV> struct Dft<T, 2, INV> {
  using C = cplx<T>;
  static __device__ __forceinline__ void run(C (&v)[2]) {
    const C t = v[0];
    v[0] = cadd(t, v[1]);
    v[1] = csub(t, v[1]);
  }
};
template <typename T, bool INV> struct Dft<T, 3, INV> {
  using C = cplx<T>;
  static __device__ __forceinline__ void run(C (&v)[3]) {
    const T s3 = T(0.86602540378443864676);
    const C s = cadd(v[1], v[2]);
    C u = rot90<C, INV>(csub(v[1], v[2]));
    u.x *= s3; u.y *= s3;
    const C t = cmk<C>(v[0].x - T(0.5) * s.x, v[0].y - T(0.5) * s.y);
    v[0] = cadd(v[0], s);
    v[1] = cadd(t, u);
    v[2] = csub(t, u);
  }
};
template <typename T, bool INV> struct Dft<T, 4, INV> {
  using C = cplx<T>;
  static __device__ __forceinline__ void run(C (&v)[4]) {
    const C a = cadd(v[0], v[2]), b = csub(v[0], v[2]), c = cadd(v[1], v[3]), d = rot90<C, INV>(csub(v[1], v[3]));
    v[0] = cadd(a, c); v[2] = csub(a, c); v[1] = cadd(b, d); v[3] = csub(b, d);
  }
};
template <typename T, bool INV> struct Dft<T, 5, INV> {
  using C = cplx<T>;
  static __device__ __forceinline__ void run(C (&v)[5]) {
    const T c1 = T(0.30901699437494742410), c2 = T(-0.80901699437494742410);
    const T s1 = T(0.95105651629515357212), s2 = T(0.58778525229247312917);
    const C s14 = cadd(v[1], v[4]), d14 = csub(v[1], v[4]), s23 = cadd(v[2], v[3]), d23 = csub(v[2], v[3]);
    const C a1 = cmk<C>(v[0].x + c1 * s14.x + c2 * s23.x, v[0].y + c1 * s14.y + c2 * s23.y);
    const C a2 = cmk<C>(v[0].x + c2 * s14.x + c1 * s23.x, v[0].y + c2 * s14.y + c1 * s23.y);
    const C b1 = rot90<C, INV>(cmk<C>(s1 * d14.x + s2 * d23.x, s1 * d14.y + s2 * d23.y));
    const C b2 = rot90<C, INV>(cmk<C>(s2 * d14.x - s1 * d23.x, s2 * d14.y - s1 * d23.y));
    v[0] = cadd(v[0], cadd(s14, s23));
    v[1] = cadd(a1, b1); v[4] = csub(a1, b1);
    v[2] = cadd(a2, b2); v[3] = csub(a2, b2);
  }
};
template <typename T, bool INV> struct Dft<T, 8, INV> {
  using C = cplx<T>;
  static __device__ __forceinline__ void run(C (&v)[8]) {
    const T r2 = T(0.70710678118654752440);
    C e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    Dft<T, 4, INV>::run(e);
    Dft<T, 4, INV>::run(o);
    C t1, t3;
    const C t2 = rot90<C, INV>(o[2]);
    if (!INV) {
      t1 = cmk<C>(r2 * (o[1].x + o[1].y), r2 * (o[1].y - o[1].x));
      t3 = cmk<C>(r2 * (o[3].y - o[3].x), -r2 * (o[3].x + o[3].y));
    } else {
      t1 = cmk<C>(r2 * (o[1].x - o[1].y), r2 * (o[1].x + o[1].y));
      t3 = cmk<C>(-r2 * (o[3].x + o[3].y), r2 * (o[3].x - o[3].y));
    }
    v[0] = cadd(e[0], o[0]); v[4] = csub(e[0], o[0]);
    v[1] = cadd(e[1], t1); v[5] = csub(e[1], t1);
    v[2] = cadd(e[2], t2); v[6] = csub(e[2], t2);
    v[3] = cadd(e[3], t3); v[7] = csub(e[3], t3);
  }
};

// Coprime factors P * Q by the prime-factor map (no twiddles): input Q i + P j, output k with
// k = ki (mod P), k = kj (mod Q). EP and EQ are the CRT idempotents.
template <typename T, int P, int Q, int EP, int EQ, bool INV> struct DftPfa {
  using C = cplx<T>;
  static __device__ __forceinline__ void run(C (&v)[P * Q]) {
    C g[P][Q];
#pragma unroll
    for (int i = 0; i < P; ++i) {
#pragma unroll
      for (int j = 0; j < Q; ++j) g[i][j] = v[(Q * i + P * j) % (P * Q)];
      Dft<T, Q, INV>::run(g[i]);
    }
#pragma unroll
    for (int j = 0; j < Q; ++j) {
      C h[P];
#pragma unroll
      for (int i = 0; i < P; ++i) h[i] = g[i][j];
      Dft<T, P, INV>::run(h);
#pragma unroll
      for (int i = 0; i < P; ++i) v[(EP * i + EQ * j) % (P * Q)] = h[i];
    }
  }
};
template <typename T, bool INV> struct Dft<T, 6, INV> : DftPfa<T, 2, 3, 3, 4, INV> {};
template <typename T, bool INV> struct Dft<T, 10, INV> : DftPfa<T, 2, 5, 5, 6, INV> {};
template <typename T, bool INV> struct Dft<T, 12, INV> : DftPfa<T, 3, 4, 4, 9, INV> {};

template <typename T, bool INV> struct Dft<T, 9, INV> {
  using C = cplx<T>;
  static __device__ __forceinline__ void run(C (&v)[9]) {
    // W9^1, W9^2, W9^4 (forward)
    const T c1 = T(0.76604444311897803520), s1 = T(0.64278760968653932632);
    const T c2 = T(0.17364817766693034885), s2 = T(0.98480775301220805937);
    const T c4 = T(-0.93969262078590838405), s4 = T(0.34202014332566873304);
    const T sg = INV ? T(1) : T(-1);
    C g[3][3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
#pragma unroll
      for (int i = 0; i < 3; ++i) g[j][i] = v[3 * i + j];
      Dft<T, 3, INV>::run(g[j]);
    }
    g[1][1] = cmul(g[1][1], cmk<C>(c1, sg * s1));
    g[1][2] = cmul(g[1][2], cmk<C>(c2, sg * s2));
    g[2][1] = cmul(g[2][1], cmk<C>(c2, sg * s2));
    g[2][2] = cmul(g[2][2], cmk<C>(c4, sg * s4));
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      C h[3] = {g[0][k], g[1][k], g[2][k]};
      Dft<T, 3, INV>::run(h);
#pragma unroll
      for (int m = 0; m < 3; ++m) v[k + 3 * m] = h[m];
    }
  }
};

template <typename T, bool INV> struct Dft<T, 16, INV> {
  using C = cplx<T>;
  static __device__ __forceinline__ void run(C (&v)[16]) {
    // W16^k, k = 1, 2, 3, 6, 9 (forward); W16^4 is a quarter turn
    const T c1 = T(0.92387953251128675613), s1 = T(0.38268343236508977173), r2 = T(0.70710678118654752440);
    const T sg = INV ? T(1) : T(-1);
    const C w1 = cmk<C>(c1, sg * s1), w2 = cmk<C>(r2, sg * r2), w3 = cmk<C>(s1, sg * c1);
    const C w6 = cmk<C>(-r2, sg * r2), w9 = cmk<C>(-c1, -sg * s1);
    C g[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
      for (int i = 0; i < 4; ++i) g[j][i] = v[4 * i + j];
      Dft<T, 4, INV>::run(g[j]);
    }
    g[1][1] = cmul(g[1][1], w1); g[1][2] = cmul(g[1][2], w2); g[1][3] = cmul(g[1][3], w3);
    g[2][1] = cmul(g[2][1], w2); g[2][2] = rot90<C, INV>(g[2][2]); g[2][3] = cmul(g[2][3], w6);
    g[3][1] = cmul(g[3][1], w3); g[3][2] = cmul(g[3][2], w6); g[3][3] = cmul(g[3][3], w9);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      C h[4] = {g[0][k], g[1][k], g[2][k], g[3][k]};
      Dft<T, 4, INV>::run(h);
#pragma unroll
      for (int m = 0; m < 4; ++m) v[k + 4 * m] = h[m];
    }
  }
};

// Factors of a line: RA points per pass-A butterfly, RB per pass-B one (the larger first: the passes
// that also touch global memory are the A passes, and a wider butterfly keeps more loads in flight).
template <int N> struct Line;
#define PGJ_LINE(N_, A_, B_)                                       \
  template <> struct Line<N_> {                                    \
    static constexpr int RA = A_, RB = B_;                         \
  };
PGJ_LINE(4, 2, 2)
PGJ_LINE(6, 3, 2)
PGJ_LINE(8, 4, 2)
PGJ_LINE(10, 5, 2)
PGJ_LINE(12, 4, 3)
PGJ_LINE(16, 4, 4)
PGJ_LINE(18, 6, 3)
PGJ_LINE(20, 5, 4)
PGJ_LINE(24, 6, 4)
PGJ_LINE(30, 6, 5)
PGJ_LINE(32, 8, 4)
PGJ_LINE(36, 6, 6)
PGJ_LINE(40, 8, 5)
PGJ_LINE(48, 8, 6)
PGJ_LINE(50, 10, 5)
PGJ_LINE(54, 9, 6)
PGJ_LINE(60, 10, 6)
PGJ_LINE(64, 8, 8)
PGJ_LINE(72, 9, 8)
PGJ_LINE(80, 10, 8)
PGJ_LINE(90, 10, 9)
PGJ_LINE(96, 12, 8)
PGJ_LINE(100, 10, 10)
PGJ_LINE(108, 12, 9)
PGJ_LINE(120, 12, 10)
PGJ_LINE(128, 16, 8)
#undef PGJ_LINE

// position of wavenumber k of a transformed line
template <int N> __device__ __forceinline__ int line_pos(int k) {
  return (k % Line<N>::RA) * Line<N>::RB + k / Line<N>::RA;
}

// pass A butterfly of offset b on v[a] = x[RB a + b]; tw: W_N^j, j < N (forward)
template <typename T, int N>
__device__ __forceinline__ void line_a(cplx<T> (&v)[Line<N>::RA], int b, const cplx<T>* tw) {
  Dft<T, Line<N>::RA, false>::run(v);
#pragma unroll
  for (int k = 1; k < Line<N>::RA; ++k) v[k] = cmul(v[k], tw[b * k]);
}
// its inverse: v[ka] at position RB ka + b
template <typename T, int N>
__device__ __forceinline__ void line_a_inv(cplx<T> (&v)[Line<N>::RA], int b, const cplx<T>* tw) {
#pragma unroll
  for (int k = 1; k < Line<N>::RA; ++k) v[k] = cmul(v[k], cconj(tw[b * k]));
  Dft<T, Line<N>::RA, true>::run(v);
}

}  // namespace pgj
