// Cluster-resident PCG: one thread-block cluster per load runs every iteration of a certified attempt
// in one launch (the recurrence of resident.py:119-131 of exp/asg_gpu_resident_20261103).
//
// Why. On small grids an iteration of separate kernels is a chain of four launches, each with a
// grid-wide reduction at its end, around very little work. The loads of a solve never exchange
// anything inside the recurrence, so one load needs no grid-wide synchronisation: a cluster of CL
// blocks (one per SM) owns it, block c the z planes [c ZC, (c + 1) ZC). Phases are separated by
// cluster barriers, sums are exchanged through distributed shared memory, and planes that a
// neighbour needs go through global memory (the L2 holds a load's vectors).
//
//   operator  q = K p over the block's ZC element planes: every element once. The forces on the
//             plane above go to the next block, those on the first row of a y tile to the tile above.
//             -> barrier: p.q and sum q, alpha
//   update    d += alpha p, r -= alpha q, s.(r - mean r) as complex pairs of real slabs, 2D DFT in
//             place, half spectra to memory -> barrier: ||r||^2, sum r; masks
//   z pass    lines along z of this block's share of the (ky, kx) columns: forward, symbol, r.z by
//             Parseval, inverse -> barrier: beta
//   inverse   half spectra to complex pairs, inverse 2D DFT, s.w -> barrier: mean(s.w)
//   direction p = (s.w - mean) + beta p, on the block's planes and its copy of the plane above
//
// FP32 recurrences also take their true-residual replacements here: d is added to the FP64 iterate,
// r = f - K x with the same operator in FP64, and the recurrence continues from T(r).
//
// What bounds it: below n = 24 the four exchanges (0.8k to 2.5k clocks each: block sum, travel, and for the
// two that order the spectra a release that waits for the block's stores), above that the element
// arithmetic and the latency of the phases' loads at 9 to 16 warps per SM. Per iteration, six loads, one
// B200, against separate kernels (pgj_planes.cuh; FP64 / mixed): n = 16 10.6 / 9.8 us against 38.6 / 47.8,
// n = 24 21.1 / 18.3, n = 32 29.4 / 23.9, n = 36 68 / 48 against 65 / 65, n = 40 100 / 65 against 71 / 69,
// n = 48 130 / 88 against 102 / 87: above n = 32 in FP64 and n = 36 in mixed precision, where p or q no longer
// fit in shared memory, the whole GPU's separate kernels win and these are not built.
//
// Vectors are held plane by plane, [z][component][y][x] per load; p is [z][y][x][component], the
// order in which the operator reads whole triples. The blocks of a cluster always take the same
// branch: every decision is formed by every thread from the same sums in the same order.
#pragma once
#include "pgj_internal.h"
#include "pgj_dft.cuh"
#include "pgj_tri.cuh"

namespace pgj {

struct ResidentArgs {
  int lpd, cap, loads;
  const double* a;        // (designs, N)
  const void* sp;         // (designs, 3, N) T: scale field by component
  const void* sym;        // (6, n, n, ns) T
  const void* tw;         // n complex T twiddles
  const double* f;        // (L, 3N) right-hand sides (FP32: true residuals)
  double* x;              // (L, 3N) FP64 iterate
  const double* r0;       // (L, 3N) certified residual
  void* r;                // (L, 3N) T recurrence residual
  void* d;                // (L, 3N) T correction
  void* p;                // (L, 3N) T direction where it does not fit in shared memory
  void* q;                // (L, 3N) T
  void* spec;             // (L, 3, n, n ns) complex T
  double* q64;            // (L, 3N) FP32: K x of a replacement
  char* halo;             // (L, resident_halo_bytes) planes handed between the blocks of a cluster
  LoadScalars* out;       // certificate records
  int* counters;          // [3]: most replacements of a load
  double rel_delta2;
  OpConst kc;
};

// One grid: CL blocks per cluster (CL divides N), TY node rows per operator tile (TY divides N), NT
// threads; PG slab pairs per transform group (all of them, or a multiple of 3 so that a group is
// whole planes), CS z-pass columns in shared memory at a time; PS / QS: p / q live in shared memory; TX:
// planes for a neighbour go straight into its shared memory.
template <int N_, typename T_, int CL_, int TY_, int NT_, int PG_, int CS_, bool PS_, bool QS_, bool TX_>
struct ResidentCfg {
  using T = T_;
  static constexpr int N = N_, CL = CL_, TY = TY_, NT = NT_, PG = PG_, CS = CS_;
  static constexpr bool PS = PS_, QS = QS_, TX = TX_;
  static constexpr int ZC = N / CL, NCH = N / TY, NW = NT / 32, NS = N / 2 + 1;
  static constexpr int PL = 3 * N * N;                 // values of one plane
  static constexpr int SL = 3 * ZC, NP = (SL + 1) / 2;  // real slabs of a block, complex pairs
  static constexpr int NG = (NP + PG - 1) / PG;
  static constexpr int PX = N + 1;                     // odd row pitch of the pair buffers
  static constexpr int M = N * NS, CM = (M + CL - 1) / CL, NSUB = (CM + CS - 1) / CS;
  static constexpr bool SWS = NG == 1;                 // s.w stays in the pair buffer until the direction
  static constexpr size_t al(size_t v) { return (v + 15) / 16 * 16; }
  static constexpr size_t mx(size_t a, size_t b) { return a > b ? a : b; }
  static constexpr size_t o_bar = 0;  // cluster barrier
  static constexpr size_t o_tw = 64;
  static constexpr size_t o_slot = al(o_tw + N * 2 * sizeof(T));
  static constexpr size_t o_bnd = al(o_slot + size_t(2 * CL + NW) * 4 * 8);
  static constexpr size_t o_p = al(o_bnd + (NCH > 1 ? size_t(ZC) * NCH * 3 * N * 8 : 0));
  static constexpr size_t o_q = al(o_p + (PS ? size_t(ZC + 1) * PL * sizeof(T) : 0));
  static constexpr size_t o_low = al(o_q + (QS ? size_t(ZC) * PL * sizeof(T) : 0));  // plane and tile rows from below
  static constexpr size_t o_u = al(o_low + (TX ? size_t(PL + (NCH > 1 ? NCH * 3 * N : 0)) * sizeof(T) : 0));
  static constexpr size_t u_fft = size_t(PG) * N * PX * 2 * sizeof(T);
  static constexpr size_t u_z = size_t(3) * N * CS * 2 * sizeof(T);
  static constexpr size_t u_x = size_t(2) * 9 * N * TY * 8;
  static constexpr size_t smem = o_u + mx(u_fft, mx(u_z, u_x));
  // halo area of one load: planes from below and their tile rows (FP64 room), s.w and p planes
  static constexpr size_t h_low = 0;
  static constexpr size_t h_bnd = h_low + size_t(CL) * PL * 8;
  static constexpr size_t h_sw = h_bnd + size_t(CL) * NCH * 3 * N * 8;
  static constexpr size_t h_p = h_sw + size_t(CL) * PL * sizeof(T);
  static constexpr size_t halo = h_p + size_t(CL) * PL * sizeof(T);
  static_assert(CL * ZC == N && TY * NCH == N && NT % 32 == 0 && N * TY <= NT && CL <= 16, "shape");
  static_assert(NG == 1 || PG % 3 == 0, "groups are whole planes");
  static_assert(!TX || QS, "s.w of the plane above arrives in the block's q planes");
  static_assert(smem <= 227 * 1024 - 1024, "shared memory");
};

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}
__device__ __forceinline__ void store_cluster(uint32_t local, unsigned rank, double v) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote) : "r"(local), "r"(rank));
  asm volatile("st.shared::cluster.f64 [%0], %1;\n" ::"r"(remote), "d"(v) : "memory");
}
__device__ __forceinline__ uint32_t cluster_addr(uint32_t local, unsigned rank) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote) : "r"(local), "r"(rank));
  return remote;
}
// Store into another block's shared memory that counts its bytes on that block's mbarrier: the reader's
// wait alone makes the value visible, no fence on either side.
__device__ __forceinline__ void store_async(uint32_t remote, double v, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];\n" ::"r"(remote),
               "l"(__double_as_longlong(v)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void store_async(uint32_t remote, float v, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];\n" ::"r"(remote),
               "r"(__float_as_uint(v)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ double xor_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Barrier over the blocks of a cluster: every block has a pair of mbarriers, used in turn, that take
// one arrival from each block of the cluster, itself included. (In turn: a block that has passed
// barrier k may arrive for k + 1 before every arrival of k has reached a third block; on one mbarrier
// that arrival would count for k there. It arrives for k + 2 only after all have passed k.) Release at cluster scope before the arrival and
// acquire in the wait order the global and shared memory traffic of the phases. The wait is bounded
// (about a second): a block that gives up marks itself dead, reports PGJ_ERR_TIMEOUT, stops arriving
// and leaves at the end of its iteration, and the others follow the same way.
struct ClusterBar {
  uint64_t bar[2];
  uint64_t tx[2];  // sums and planes that arrive by asynchronous stores: operator, s.w (in turn, as above)
  int dead;
};
constexpr long long kClusterWaitClocks = 2000000000ll;

template <int CL>
__device__ __forceinline__ void cluster_arrive(ClusterBar* b, unsigned phase) {  // by threads t < CL, after a block barrier
  if (threadIdx.x < CL && !*(volatile int*)&b->dead) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n"
                 : "=r"(remote)
                 : "r"(smem_u32(&b->bar[phase & 1u])), "r"(threadIdx.x));
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(remote) : "memory");
  }
}
__device__ __forceinline__ void cluster_wait_on(ClusterBar* b, uint64_t* which, unsigned parity,
                                                long long limit = kClusterWaitClocks) {
  volatile int* dead = &b->dead;
  const uint32_t at = smem_u32(which);
  const long long t0 = clock64();
  for (int tries = 0; tries < (1 << 28); ++tries) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(at), "r"(parity)
        : "memory");
    if (ok || *dead) break;
    if (clock64() - t0 > limit) {
      *dead = 1;
      break;
    }
  }
}
__device__ __forceinline__ void cluster_wait(ClusterBar* b, unsigned& phase) {
  cluster_wait_on(b, &b->bar[phase & 1u], (phase >> 1) & 1u);
  ++phase;
}
template <int CL>
__device__ __forceinline__ void cluster_sync_all(ClusterBar* b, unsigned& phase) {
  __syncthreads();
  cluster_arrive<CL>(b, phase);
  cluster_wait(b, phase);
}

// Cluster-wide sums of K values per thread, in two halves so that work that does not need the sums
// can run while they travel. publish: the block's sums (warps in order) go from warp 0 to a slot of
// every block, followed by the arrival. collect: after the wait every warp adds the slots in the same
// order, so all threads of the cluster end with the same bits. Two slot sets alternate over the
// barriers: a fast block never overwrites what a slow one still reads. (Every warp writing to every
// block instead cost NW times the packets: 2.8k against 1.3k clocks a barrier at n = 16.)
// ASYNC: the sums travel as asynchronous stores and the reader waits for their bytes, together with
// `more` bytes that the other blocks store into this one before their publish. Nothing in global memory
// is ordered by that form (a release waits for every store under way: 1.7k clocks at n = 16).
template <class Cfg, int K, bool ASYNC>
__device__ __forceinline__ void cluster_publish(double (&v)[K], double* wsum, double* slots, unsigned rank,
                                                ClusterBar* bar, unsigned phase, uint64_t* tx, unsigned more) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < K; ++k) v[k] = xor_sum(v[k]);
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < K; ++k) wsum[warp * 4 + k] = v[k];
  __syncthreads();
  if (warp == 0) {
    if (ASYNC && lane == 0) mbar_expect_tx(tx, unsigned(Cfg::CL * K * 8) + more);
    double t[K];
#pragma unroll
    for (int k = 0; k < K; ++k) t[k] = xor_sum(lane < Cfg::NW ? wsum[lane * 4 + k] : 0.0);
    if (lane < Cfg::CL && !*(volatile int*)&bar->dead) {
      const uint32_t at = smem_u32(slots + rank * 4);
      if constexpr (ASYNC) {
        const uint32_t to = cluster_addr(at, unsigned(lane)), tb = cluster_addr(smem_u32(tx), unsigned(lane));
#pragma unroll
        for (int k = 0; k < K; ++k) store_async(to + 8 * k, t[k], tb);
      } else {
#pragma unroll
        for (int k = 0; k < K; ++k) store_cluster(at + 8 * k, unsigned(lane), t[k]);
      }
    }
    if constexpr (!ASYNC) {
      __syncwarp();
      cluster_arrive<Cfg::CL>(bar, phase);
    }
  }
}
template <class Cfg, int K, bool ASYNC>
__device__ __forceinline__ void cluster_collect(double (&v)[K], const double* slots, ClusterBar* bar, unsigned& phase,
                                                uint64_t* tx, unsigned& tphase) {
  const int lane = threadIdx.x & 31;
  if constexpr (ASYNC) {
    cluster_wait_on(bar, tx, tphase);
    tphase ^= 1u;
  } else {
    cluster_wait(bar, phase);
  }
#pragma unroll
  for (int k = 0; k < K; ++k) v[k] = xor_sum(lane < Cfg::CL ? slots[lane * 4 + k] : 0.0);
}

// K(a) over the block's ZC element planes (z0 .. z0 + ZC - 1), in the arithmetic type R. node(j, y, x)
// is the triple of node plane z0 + j, j <= ZC. put(s, y, x, q): forces of these elements on node plane
// z0 + s, s <= ZC; with several y tiles the first row of a tile lacks the tile below, which comes as
// bnd(s, tile, x, q). dot: adds u.q and sum q of everything put.
template <class Cfg, typename R, class Node, class Put, class Bnd>
__device__ __forceinline__ void slab_operator(const double* __restrict__ a, const OpConst& kc, R* xch, Node node,
                                              Put put, Bnd bnd, bool dot, double (&acc)[4]) {
  constexpr int N = Cfg::N, TY = Cfg::TY, ZC = Cfg::ZC, NCH = Cfg::NCH, NE = N * TY;
  const int tid = threadIdx.x;
  const bool on = tid < NE;
  const int ty = tid / N, x = tid - ty * N;
  const int xp = x + 1 == N ? 0 : x + 1, xl = x == 0 ? N - 1 : x - 1;
  const int tl = ty * N + xl;                                  // element to the left
  const int tb = (ty == 0 ? TY - 1 : ty - 1) * N;              // row of elements below (NCH == 1: periodic)
  int par = 0;
#pragma unroll 1
  for (int ch = 0; ch < NCH; ++ch) {
    const int y = ch * TY + ty, yp = y + 1 == N ? 0 : y + 1;
    Tri<R> F0[4], Up[4];
    auto face = [&](int j, Tri<R> (&F)[4]) {
      const Tri<R> u00 = node(j, y, x), u10 = node(j, y, xp), u01 = node(j, yp, x), u11 = node(j, yp, xp);
      const Tri<R> sx0 = u10 + u00, dx0 = u10 - u00, sx1 = u11 + u01, dx1 = u11 - u01;
      F[0] = sx1 + sx0;
      F[1] = dx1 + dx0;
      F[2] = sx1 - sx0;
      F[3] = dx1 - dx0;
    };
    const double* ap = a + y * N + x;
    double an = 0.0;
    if (on) {
      an = __ldg(ap);
      face(0, F0);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) Up[k] = Tri<R>::make(R(0), R(0), R(0));
#pragma unroll(ZC <= 2 ? ZC + 1 : 1)
    for (int s = 0; s <= ZC; ++s) {
      R* xb = xch + par * 9 * NE;
      par ^= 1;
      Tri<R> c00, c01;
      if (on) {
        Tri<R> G[4];
        if (s < ZC) {
          const R ae = R(an);
          if (s + 1 < ZC) an = __ldg(ap + (s + 1) * N * N);
          Tri<R> F1[4];
          face(s + 1, F1);
          R Q[8][3], P[8][3];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const Tri<R> sum = F1[k] + F0[k], dif = F1[k] - F0[k];
#pragma unroll
            for (int c = 0; c < 3; ++c) { Q[k][c] = sum.get(c); Q[k + 4][c] = dif.get(c); }
            F0[k] = F1[k];
          }
          element_modal<R>(Q, ae, kc, P);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const Tri<R> lo = Tri<R>::make(P[k][0], P[k][1], P[k][2]);
            const Tri<R> hi = Tri<R>::make(P[k + 4][0], P[k + 4][1], P[k + 4][2]);
            G[k] = (lo - hi) + Up[k];
            Up[k] = lo + hi;
          }
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k) G[k] = Up[k];
        }
        // corners of the face: (x, y) stays, (x+1, y), (x, y+1), (x+1, y+1) go to their owners
        const Tri<R> ly0 = G[0] - G[2], ly1 = G[1] - G[3], uy0 = G[0] + G[2], uy1 = G[1] + G[3];
        c00 = ly0 - ly1;
        c01 = uy0 - uy1;
        (ly0 + ly1).store(xb + (0 * NE + tid) * 3);
        c01.store(xb + (1 * NE + tid) * 3);
        (uy0 + uy1).store(xb + (2 * NE + tid) * 3);
      }
      __syncthreads();  // corners published; the other half of xch is free again
      if (on) {
        Tri<R> q = c00 + Tri<R>::load(xb + (0 * NE + tl) * 3);
        if (NCH == 1 || ty >= 1)
          q = (q + Tri<R>::load(xb + (1 * NE + tb + x) * 3)) + Tri<R>::load(xb + (2 * NE + tb + xl) * 3);
        put(s, y, x, q);
        if (dot) {
          const Tri<R> u = node(s, y, x);
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            acc[0] += double(u.get(c)) * double(q.get(c));
            acc[1 + c] += double(q.get(c));
          }
        }
        if (NCH > 1 && ty == TY - 1) {
          const Tri<R> b = c01 + Tri<R>::load(xb + (2 * NE + tl) * 3);
          bnd(s, ch + 1 == NCH ? 0 : ch + 1, x, b);
          if (dot) {
            const Tri<R> u = node(s, yp, x);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              acc[0] += double(u.get(c)) * double(b.get(c));
              acc[1 + c] += double(b.get(c));
            }
          }
        }
      }
    }
  }
}

template <class Cfg>
__global__ void __launch_bounds__(Cfg::NT, 1) k_resident_pcg(const ResidentArgs A) {
  using T = typename Cfg::T;
  using C = cplx<T>;
  constexpr int N = Cfg::N, CL = Cfg::CL, ZC = Cfg::ZC, NT = Cfg::NT, NS = Cfg::NS, PL = Cfg::PL, SL = Cfg::SL;
  constexpr int PG = Cfg::PG, NG = Cfg::NG, NP = Cfg::NP, PX = Cfg::PX, M = Cfg::M, CM = Cfg::CM, CS = Cfg::CS;
  constexpr int RA = Line<N>::RA, RB = Line<N>::RB, NN = N * N, TY = Cfg::TY, NCH = Cfg::NCH;
  constexpr size_t NV = size_t(NN) * N, N3 = 3 * NV;
  constexpr bool TX = Cfg::TX;
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x;
  const unsigned rank = cluster_rank();
  const int load = blockIdx.x / CL;
  LoadScalars& O = A.out[load];
  // masks of the attempt (resident.py:120); the same record for every block of the cluster
  int it = O.iterations, bad = O.bad;
  const double target2 = O.target2;
  bool active = O.res2 > target2 && it < A.cap && !bad && !O.frozen;
  if (!active) return;
  const double rel_delta2 = sizeof(T) == 4 ? A.rel_delta2 : 0.0;
  double anchor = O.res2, rz = 0.0;
  double mr[3] = {O.mean_r[0], O.mean_r[1], O.mean_r[2]};
  int reps = 0;

  ClusterBar* bar = reinterpret_cast<ClusterBar*>(smem + Cfg::o_bar);
  unsigned phase = 0, tphase0 = 0, tphase1 = 0;
  if (tid == 0) {
    mbar_init(&bar->bar[0], CL);
    mbar_init(&bar->bar[1], CL);
    mbar_init(&bar->tx[0], 1);
    mbar_init(&bar->tx[1], 1);
    fence_mbar_init();
    bar->dead = 0;
  }
  C* tw = reinterpret_cast<C*>(smem + Cfg::o_tw);
  double* slot0 = reinterpret_cast<double*>(smem + Cfg::o_slot);
  double* slot1 = slot0 + CL * 4;
  double* wsum = slot1 + CL * 4;
  C* buf = reinterpret_cast<C*>(smem + Cfg::o_u);  // pair buffers / z lines / corner exchange
  const int z0 = int(rank) * ZC;
  const unsigned up = rank + 1 == CL ? 0u : rank + 1;
  const size_t off = size_t(load) * N3 + size_t(z0) * PL;  // this block's planes, any vector
  T* r = static_cast<T*>(A.r) + off;
  T* d = static_cast<T*>(A.d) + off;
  char* halo = A.halo + size_t(load) * Cfg::halo;
  double* hlow = reinterpret_cast<double*>(halo + Cfg::h_low);  // FP64 room, holds T or double
  double* hbnd = reinterpret_cast<double*>(halo + Cfg::h_bnd);
  T* hsw = reinterpret_cast<T*>(halo + Cfg::h_sw);
  T* p_own = Cfg::PS ? reinterpret_cast<T*>(smem + Cfg::o_p) : static_cast<T*>(A.p) + off;
  T* p_top = Cfg::PS ? p_own + ZC * PL : reinterpret_cast<T*>(halo + Cfg::h_p) + size_t(rank) * PL;
  T* q = Cfg::QS ? reinterpret_cast<T*>(smem + Cfg::o_q) : static_cast<T*>(A.q) + off;
  // TX: where this block's values for the plane above go, and where its own from below arrive
  T* low_in = reinterpret_cast<T*>(smem + Cfg::o_low);
  const uint32_t up_low = TX ? cluster_addr(smem_u32(low_in), up) : 0u;
  const unsigned down = rank == 0 ? unsigned(CL - 1) : rank - 1;
  T* sw_in = reinterpret_cast<T*>(smem + Cfg::o_q);  // s.w of the plane above (q is free by then)
  const uint32_t down_sw = TX ? cluster_addr(smem_u32(sw_in), down) : 0u;
  const uint32_t up_tx = TX ? cluster_addr(smem_u32(&bar->tx[0]), up) : 0u;
  const uint32_t down_tx = TX ? cluster_addr(smem_u32(&bar->tx[1]), down) : 0u;
  C* spec = static_cast<C*>(A.spec) + size_t(load) * 3 * N * M;
  const size_t dsg = size_t(load / A.lpd);
  const T* sc = static_cast<const T*>(A.sp) + dsg * N3 + size_t(z0) * NN;  // + c NV + (z - z0) NN
  const double* a = A.a + dsg * NV + size_t(z0) * NN;
  const T* sym = static_cast<const T*>(A.sym);

  for (int i = tid; i < N; i += NT) tw[i] = static_cast<const C*>(A.tw)[i];
  // r = T(certified residual), plane by plane through shared memory
  {
    T* st = reinterpret_cast<T*>(buf);
    constexpr int PB = int((Cfg::smem - Cfg::o_u) / (PL * sizeof(T)));  // planes staged at a time
    static_assert(PB >= 1, "a plane fits");
    const double* r0 = A.r0 + off;
    for (int zb = 0; zb < ZC; zb += PB) {
      const int nz = min(PB, ZC - zb);
      __syncthreads();
      for (int i = tid; i < nz * PL; i += NT) {
        const int z = i / PL, e = i - z * PL, node = e / 3, c = e - 3 * node;
        st[z * PL + c * NN + node] = T(r0[size_t(zb) * PL + i]);
      }
      __syncthreads();
      for (int i = tid; i < nz * PL; i += NT) {
        r[size_t(zb) * PL + i] = st[i];
        d[size_t(zb) * PL + i] = T(0);
      }
    }
  }
  // once, before any block reaches into another: all are running, all mbarriers initialised
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release;\n barrier.cluster.wait.acquire;\n" ::: "memory");

  // r and s of this thread's columns, loaded while the operator's sums travel where they fit
  constexpr int CPT = (NN + NT - 1) / NT;
  constexpr bool PRE = NG == 1 && CPT * SL * 2 * int(sizeof(T)) <= 224;
  T rv[PRE ? CPT * SL : 1], sv[PRE ? CPT * SL : 1];
  auto load_rs = [&]() {
    if constexpr (PRE) {
#pragma unroll
      for (int h = 0; h < CPT; ++h) {
        const int i = tid + h * NT;
#pragma unroll
        for (int sl = 0; sl < SL; ++sl) {
          rv[h * SL + sl] = i < NN ? r[sl * NN + i] : T(0);
          sv[h * SL + sl] = i < NN ? __ldg(sc + size_t(sl % 3) * NV + (sl / 3) * NN + i) : T(0);
        }
      }
    }
  };
  bool first = true;   // the first direction: p = z
  bool plain = true;   // transform r as it stands (start, replacement) instead of updating it
  double alpha = 0.0, mp[3] = {mr[0], mr[1], mr[2]};
  for (;;) {
    if (!plain) {
      // ------------------------------------------------------------------------ operator
      double acc[4] = {0.0, 0.0, 0.0, 0.0};
      T* low = reinterpret_cast<T*>(hlow) + size_t(up) * PL;
      T* lowb = reinterpret_cast<T*>(hbnd) + size_t(up) * NCH * 3 * N;
      T* bnd = reinterpret_cast<T*>(smem + Cfg::o_bnd);
      slab_operator<Cfg, T>(
          a, A.kc, reinterpret_cast<T*>(buf),
          [&](int j, int y, int x) {
            const T* pl = j < ZC ? p_own + j * PL : p_top;
            return Tri<T>::load(pl + 3 * (y * N + x));
          },
          [&](int s, int y, int x, const Tri<T>& v) {
            if (s < ZC || !TX) {
              T* o = (s < ZC ? q + s * PL : low) + y * N + x;
#pragma unroll
              for (int c = 0; c < 3; ++c) o[c * NN] = v.get(c);
            } else {
#pragma unroll
              for (int c = 0; c < 3; ++c)
                store_async(up_low + unsigned((c * NN + y * N + x) * sizeof(T)), v.get(c), up_tx);
            }
          },
          [&](int s, int t, int x, const Tri<T>& v) {
            if (s < ZC || !TX) {
              T* o = (s < ZC ? bnd + s * NCH * 3 * N : lowb) + t * 3 * N + x;
#pragma unroll
              for (int c = 0; c < 3; ++c) o[c * N] = v.get(c);
            } else {
#pragma unroll
              for (int c = 0; c < 3; ++c)
                store_async(up_low + unsigned((PL + t * 3 * N + c * N + x) * sizeof(T)), v.get(c), up_tx);
            }
          },
          true, acc);
      cluster_publish<Cfg, 4, TX>(acc, wsum, slot0, rank, bar, phase, &bar->tx[0],
                                  unsigned(PL + (NCH > 1 ? NCH * 3 * N : 0)) * unsigned(sizeof(T)));
      load_rs();
      cluster_collect<Cfg, 4, TX>(acc, slot0, bar, phase, &bar->tx[0], tphase0);
      const bool valid = isfinite(acc[0]) && acc[0] > 0.0 && isfinite(rz) && rz > 0.0;
      alpha = valid ? rz / acc[0] : 0.0;
      bad |= valid ? 0 : 1;
      // mean of r after the update (the projection of the next preconditioner input)
#pragma unroll
      for (int c = 0; c < 3; ++c) mp[c] = mr[c] - alpha * (acc[1 + c] / double(NV));
    } else {
      load_rs();
#pragma unroll
      for (int c = 0; c < 3; ++c) mp[c] = mr[c];
    }
    // ---------------------------------------------------- update and forward x/y transforms
    double sum[4] = {0.0, 0.0, 0.0, 0.0};
    {
      const T al = T(alpha);
      const T m[3] = {T(mp[0]), T(mp[1]), T(mp[2])};
      const T* low = reinterpret_cast<const T*>(hlow) + size_t(rank) * PL;
      const T* lowb = reinterpret_cast<const T*>(hbnd) + size_t(rank) * NCH * 3 * N;
      const T* bnd = reinterpret_cast<const T*>(smem + Cfg::o_bnd);
#pragma unroll 1
      for (int g = 0; g < NG; ++g) {
        const int zg = NG == 1 ? 0 : g * (2 * PG / 3);  // first plane of the group
        // r' = r - alpha q with the parts of q the neighbours computed; returns s (r' - mean r')
        auto update = [&](int z, int c, int i, int y, int x, T rk, T sk) -> T {
          if (!plain) {
            const int e = (z * 3 + c) * NN + i;
            T qv = q[e];
            if (NCH > 1 && y % TY == 0) qv += bnd[((z * NCH + y / TY) * 3 + c) * N + x];
            if (z == 0) {
              T lv = TX ? low_in[c * NN + i] : __ldcg(low + c * NN + i);
              if (NCH > 1 && y % TY == 0) {
                const int t = ((y / TY) * 3 + c) * N + x;
                lv += TX ? low_in[PL + t] : __ldcg(lowb + t);
              }
              qv += lv;
            }
            rk = rk - al * qv;
            r[e] = rk;
            const double rd = double(rk);
            sum[0] += rd * rd;
            sum[1 + c] += rd;
          }
          return sk * (rk - m[c]);
        };
        if constexpr (PRE) {
#pragma unroll
          for (int h = 0; h < CPT; ++h) {
            const int i = tid + h * NT, y = i / N, x = i - y * N;
            if (i >= NN) continue;
#pragma unroll
            for (int j = 0; j < NP; ++j) {
              const int s0 = 2 * j, s1 = s0 + 1;
              const T v0 = update(s0 / 3, s0 % 3, i, y, x, rv[h * SL + s0], sv[h * SL + s0]);
              const T v1 = s1 < SL ? update(s1 / 3, s1 % 3, i, y, x, rv[h * SL + (s1 < SL ? s1 : 0)], sv[h * SL + (s1 < SL ? s1 : 0)]) : T(0);
              buf[(j * N + y) * PX + x] = cmk<C>(v0, v1);
            }
          }
        } else {
          constexpr int UB = sizeof(T) == 8 ? 6 : 12;  // slabs whose loads are in flight together
#pragma unroll 1
          for (int i = tid; i < NN; i += NT) {
            const int y = i / N, x = i - y * N;
#pragma unroll
            for (int b = 0; b < 2 * PG; b += UB) {
              T rb[UB], sb[UB];
#pragma unroll
              for (int k = 0; k < UB; ++k) {
                const int sl = b + k, c = sl % 3, z = zg + sl / 3;
                rb[k] = sb[k] = T(0);
                if (sl >= 2 * PG || z >= ZC) continue;
                rb[k] = r[(z * 3 + c) * NN + i];
                sb[k] = __ldg(sc + size_t(c) * NV + z * NN + i);
              }
#pragma unroll
              for (int k = 0; k < UB; ++k) {
                const int sl = b + k, c = sl % 3, z = zg + sl / 3;
                if (sl < 2 * PG && z < ZC) rb[k] = update(z, c, i, y, x, rb[k], sb[k]);
              }
#pragma unroll
              for (int k = 0; k < UB; k += 2)
                if (b + k < 2 * PG) buf[(((b + k) / 2) * N + y) * PX + x] = cmk<C>(rb[k], rb[k + 1]);
            }
          }
        }
        __syncthreads();
        // x lines (y fastest over the lanes: the odd pitch keeps them on distinct banks)
        for (int w = tid; w < PG * RB * N; w += NT) {
          const int l = w % N, t = w / N, b = t % RB, j = t / RB;
          C* at = buf + (j * N + l) * PX + b;
          C v[RA];
#pragma unroll
          for (int k = 0; k < RA; ++k) v[k] = at[RB * k];
          line_a<T, N>(v, b, tw);
#pragma unroll
          for (int k = 0; k < RA; ++k) at[RB * k] = v[k];
        }
        __syncthreads();
        for (int w = tid; w < PG * RA * N; w += NT) {
          const int l = w % N, t = w / N, ka = t % RA, j = t / RA;
          C* at = buf + (j * N + l) * PX + RB * ka;
          C v[RB];
#pragma unroll
          for (int k = 0; k < RB; ++k) v[k] = at[k];
          Dft<T, RB, false>::run(v);
#pragma unroll
          for (int k = 0; k < RB; ++k) at[k] = v[k];
        }
        __syncthreads();
        // y lines (x fastest)
        for (int w = tid; w < PG * RB * N; w += NT) {
          const int l = w % N, t = w / N, b = t % RB, j = t / RB;
          C* at = buf + (j * N + b) * PX + l;
          C v[RA];
#pragma unroll
          for (int k = 0; k < RA; ++k) v[k] = at[RB * k * PX];
          line_a<T, N>(v, b, tw);
#pragma unroll
          for (int k = 0; k < RA; ++k) at[RB * k * PX] = v[k];
        }
        __syncthreads();
        for (int w = tid; w < PG * RA * N; w += NT) {
          const int l = w % N, t = w / N, ka = t % RA, j = t / RA;
          C* at = buf + (j * N + RB * ka) * PX + l;
          C v[RB];
#pragma unroll
          for (int k = 0; k < RB; ++k) v[k] = at[k * PX];
          Dft<T, RB, false>::run(v);
#pragma unroll
          for (int k = 0; k < RB; ++k) at[k * PX] = v[k];
        }
        __syncthreads();
        // pair -> two half spectra: A = (Z(k) + conj Z(-k)) / 2, B = (Z(k) - conj Z(-k)) / 2i
        for (int w = tid; w < PG * M; w += NT) {
          const int j = w / M, k = w - j * M, ky = k / NS, kx = k - ky * NS;
          const int s0 = 2 * j, za = zg + s0 / 3, zb = zg + (s0 + 1) / 3;
          if (za >= ZC) continue;
          const C* pb = buf + j * N * PX;
          const C zk = pb[line_pos<N>(ky) * PX + line_pos<N>(kx)];
          const C zn = pb[line_pos<N>(ky == 0 ? 0 : N - ky) * PX + line_pos<N>(kx == 0 ? 0 : N - kx)];
          spec[(size_t(s0 % 3) * N + z0 + za) * M + k] = cmk<C>(T(0.5) * (zk.x + zn.x), T(0.5) * (zk.y - zn.y));
          if (zb < ZC)
            spec[(size_t((s0 + 1) % 3) * N + z0 + zb) * M + k] = cmk<C>(T(0.5) * (zk.y + zn.y), T(0.5) * (zn.x - zk.x));
        }
        if (NG > 1) __syncthreads();
      }
    }
    if (!plain) {
      cluster_publish<Cfg, 4, false>(sum, wsum, slot1, rank, bar, phase, nullptr, 0u);
      {  // the correction is not needed before the next replacement: it moves while the sums travel
        const T al = T(alpha);
        for (int i = tid; i < NN; i += NT)
#pragma unroll
          for (int sl = 0; sl < SL; ++sl) d[sl * NN + i] += al * p_own[(sl / 3) * PL + 3 * i + sl % 3];
      }
      cluster_collect<Cfg, 4, false>(sum, slot1, bar, phase, nullptr, tphase0);
      // the bookkeeping of the reference's update (masks, latch, cap); bad holds the operator's verdict
      const double res2 = sum[0];
      const bool valid = !bad, finite = isfinite(res2);
      ++it;
      const bool keep = valid && finite && res2 > target2 && it < A.cap;
      bad |= finite ? 0 : 1;
      active = keep;
#pragma unroll
      for (int c = 0; c < 3; ++c) mr[c] = sum[1 + c] / double(NV);
      if constexpr (sizeof(T) == 4) {
        const bool ok = valid && finite && it < A.cap;
        if (rel_delta2 > 0.0 && ok && ((keep && res2 < rel_delta2 * anchor) || (!keep && res2 <= target2))) {
          // ------------------------------------------------ true-residual replacement (FP64)
          ++reps;
          __syncthreads();  // d as every thread of the block left it
          double* x = A.x + off;
          for (int i = tid; i < ZC * NN; i += NT) {
            const int z = i / NN, e = i - z * NN;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              x[3 * size_t(i) + c] += double(d[(z * 3 + c) * NN + e]);
              d[(z * 3 + c) * NN + e] = T(0);
            }
          }
          cluster_sync_all<CL>(bar, phase);  // x of every block
          const double* xt = A.x + size_t(load) * N3 + size_t(up) * ZC * PL;  // the plane above
          double* q64 = A.q64 + off;
          double* b64 = reinterpret_cast<double*>(smem + Cfg::o_bnd);
          double none[4] = {0.0, 0.0, 0.0, 0.0};
          slab_operator<Cfg, double>(
              a, A.kc, reinterpret_cast<double*>(buf),
              [&](int j, int y, int xx) {
                if (j < ZC) return Tri<double>::load(x + size_t(j) * PL + 3 * (y * N + xx));
                const double* g = xt + 3 * (y * N + xx);
                return Tri<double>::make(__ldcg(g), __ldcg(g + 1), __ldcg(g + 2));
              },
              [&](int s, int y, int xx, const Tri<double>& v) {
                double* o = (s < ZC ? q64 + size_t(s) * PL : hlow + size_t(up) * PL) + y * N + xx;
#pragma unroll
                for (int c = 0; c < 3; ++c) o[c * NN] = v.get(c);
              },
              [&](int s, int t, int xx, const Tri<double>& v) {
                double* o = (s < ZC ? b64 + s * NCH * 3 * N : hbnd + size_t(up) * NCH * 3 * N) + t * 3 * N + xx;
#pragma unroll
                for (int c = 0; c < 3; ++c) o[c * N] = v.get(c);
              },
              false, none);
          cluster_sync_all<CL>(bar, phase);  // forces on the first plane, from the block below
          double rs[4] = {0.0, 0.0, 0.0, 0.0};
          const double* f = A.f + off;
          const double* low = hlow + size_t(rank) * PL;
          const double* lowb = hbnd + size_t(rank) * NCH * 3 * N;
          for (int i = tid; i < ZC * NN; i += NT) {
            const int z = i / NN, e = i - z * NN, y = e / N, xx = e - y * N;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              double qv = q64[(z * 3 + c) * NN + e];
              if (NCH > 1 && y % TY == 0) qv += b64[((z * NCH + y / TY) * 3 + c) * N + xx];
              if (z == 0) {
                double lv = __ldcg(low + c * NN + e);
                if (NCH > 1 && y % TY == 0) lv += __ldcg(lowb + ((y / TY) * 3 + c) * N + xx);
                qv += lv;
              }
              const double rv = f[3 * size_t(i) + c] - qv;
              r[(z * 3 + c) * NN + e] = T(rv);
              rs[0] += rv * rv;
              rs[1 + c] += rv;
            }
          }
          cluster_publish<Cfg, 4, false>(rs, wsum, slot0, rank, bar, phase, nullptr, 0u);
          cluster_collect<Cfg, 4, false>(rs, slot0, bar, phase, nullptr, tphase0);
          anchor = rs[0];
#pragma unroll
          for (int c = 0; c < 3; ++c) mr[c] = rs[1 + c] / double(NV);
          active = isfinite(rs[0]) && rs[0] > target2 && it < A.cap && !bad;
          if (active) {
            plain = true;  // transform the new residual; the direction is kept
            continue;
          }
        }
      }
      if (!active) break;
    } else {
      cluster_sync_all<CL>(bar, phase);  // spectra of every block
    }
    // ---------------------------------------------------------------------------- z pass
    double pv[1] = {0.0};
#pragma unroll 1
    for (int sub = 0; sub < Cfg::NSUB; ++sub) {
      const int m0 = int(rank) * CM + sub * CS;
      const int cnt = min(min(CS, CM - sub * CS), M - m0);
      if (sub > 0) __syncthreads();
      for (int w = tid; w < 3 * RB * CS; w += NT) {
        const int ml = w % CS, t = w / CS, b = t % RB, c = t / RB;
        if (ml >= cnt) continue;
        const C* src = spec + (size_t(c) * N + b) * M + m0 + ml;
        C v[RA];
#pragma unroll
        for (int k = 0; k < RA; ++k) v[k] = __ldcg(src + size_t(RB * k) * M);
        line_a<T, N>(v, b, tw);
        C* dst = buf + (c * N + b) * CS + ml;
#pragma unroll
        for (int k = 0; k < RA; ++k) dst[RB * k * CS] = v[k];
      }
      __syncthreads();
      for (int w = tid; w < RA * CS; w += NT) {
        const int ml = w % CS, ka = w / CS;
        if (ml >= cnt) continue;
        const int mm = m0 + ml, kx = mm % NS;
        const double wgt = (kx == 0 || kx == N / 2) ? 1.0 : 2.0;
        C* at = buf + RB * ka * CS + ml;
        C v[3][RB];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
#pragma unroll
          for (int k = 0; k < RB; ++k) v[c][k] = at[(c * N + k) * CS];
          Dft<T, RB, false>::run(v[c]);
        }
        double acc = 0.0;
#pragma unroll
        for (int k = 0; k < RB; ++k) {
          const size_t kk = size_t(ka + RA * k) * M + mm;
          const T c0 = __ldg(sym + kk), c1 = __ldg(sym + size_t(1) * N * M + kk), c2 = __ldg(sym + size_t(2) * N * M + kk);
          const T c3 = __ldg(sym + size_t(3) * N * M + kk), c4 = __ldg(sym + size_t(4) * N * M + kk);
          const T c5 = __ldg(sym + size_t(5) * N * M + kk);
          const C vx = v[0][k], vy = v[1][k], vz = v[2][k];
          const C wx = cmk<C>(c0 * vx.x + c3 * vy.x + c4 * vz.x, c0 * vx.y + c3 * vy.y + c4 * vz.y);
          const C wy = cmk<C>(c3 * vx.x + c1 * vy.x + c5 * vz.x, c3 * vx.y + c1 * vy.y + c5 * vz.y);
          const C wz = cmk<C>(c4 * vx.x + c5 * vy.x + c2 * vz.x, c4 * vx.y + c5 * vy.y + c2 * vz.y);
          acc += double(vx.x) * wx.x + double(vx.y) * wx.y + double(vy.x) * wy.x + double(vy.y) * wy.y +
                 double(vz.x) * wz.x + double(vz.y) * wz.y;
          v[0][k] = wx; v[1][k] = wy; v[2][k] = wz;
        }
        pv[0] += wgt * acc;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          Dft<T, RB, true>::run(v[c]);
#pragma unroll
          for (int k = 0; k < RB; ++k) at[(c * N + k) * CS] = v[c][k];
        }
      }
      __syncthreads();
      for (int w = tid; w < 3 * RB * CS; w += NT) {
        const int ml = w % CS, t = w / CS, b = t % RB, c = t / RB;
        if (ml >= cnt) continue;
        const C* src = buf + (c * N + b) * CS + ml;
        C v[RA];
#pragma unroll
        for (int k = 0; k < RA; ++k) v[k] = src[RB * k * CS];
        line_a_inv<T, N>(v, b, tw);
        C* dst = spec + (size_t(c) * N + b) * M + m0 + ml;
#pragma unroll
        for (int k = 0; k < RA; ++k) dst[size_t(RB * k) * M] = v[k];
      }
    }
    cluster_publish<Cfg, 1, false>(pv, wsum, slot0, rank, bar, phase, nullptr, 0u);
    cluster_collect<Cfg, 1, false>(pv, slot0, bar, phase, nullptr, tphase0);
    const double beta64 = first ? 0.0 : pv[0] / (rz != 0.0 ? rz : 1.0);
    rz = pv[0];
    // ------------------------------------------------------------- inverse x/y transforms, s.w
    double ms[3] = {0.0, 0.0, 0.0};
    T* swg = static_cast<T*>(A.q) + off;  // s.w where several groups share the pair buffer (q is free)
#pragma unroll 1
    for (int g = 0; g < NG; ++g) {
      const int zg = NG == 1 ? 0 : g * (2 * PG / 3);
      if (g > 0) __syncthreads();
      constexpr int UF = sizeof(T) == 8 ? 4 : 6;  // points whose loads are in flight together
#pragma unroll 1
      for (int w0 = tid; w0 < PG * M; w0 += UF * NT) {
        C va[UF], vb[UF];
#pragma unroll
        for (int u = 0; u < UF; ++u) {
          const int w = w0 + u * NT, j = w / M, k = w - j * M;
          const int s0 = 2 * j, za = zg + s0 / 3, zb = zg + (s0 + 1) / 3;
          va[u] = vb[u] = cmk<C>(T(0), T(0));
          if (w >= PG * M || za >= ZC) continue;
          va[u] = __ldcg(spec + (size_t(s0 % 3) * N + z0 + za) * M + k);
          if (zb < ZC) vb[u] = __ldcg(spec + (size_t((s0 + 1) % 3) * N + z0 + zb) * M + k);
        }
#pragma unroll
        for (int u = 0; u < UF; ++u) {
          const int w = w0 + u * NT, j = w / M, k = w - j * M, ky = k / NS, kx = k - ky * NS;
          if (w >= PG * M) continue;
          C* pb = buf + j * N * PX;
          pb[line_pos<N>(ky) * PX + line_pos<N>(kx)] = cmk<C>(va[u].x - vb[u].y, va[u].y + vb[u].x);
          if (kx != 0 && kx != N / 2)
            pb[line_pos<N>(ky == 0 ? 0 : N - ky) * PX + line_pos<N>(N - kx)] =
                cmk<C>(va[u].x + vb[u].y, vb[u].x - va[u].y);
        }
      }
      __syncthreads();
      for (int w = tid; w < PG * RA * N; w += NT) {
        const int l = w % N, t = w / N, ka = t % RA, j = t / RA;
        C* at = buf + (j * N + RB * ka) * PX + l;
        C v[RB];
#pragma unroll
        for (int k = 0; k < RB; ++k) v[k] = at[k * PX];
        Dft<T, RB, true>::run(v);
#pragma unroll
        for (int k = 0; k < RB; ++k) at[k * PX] = v[k];
      }
      __syncthreads();
      for (int w = tid; w < PG * RB * N; w += NT) {
        const int l = w % N, t = w / N, b = t % RB, j = t / RB;
        C* at = buf + (j * N + b) * PX + l;
        C v[RA];
#pragma unroll
        for (int k = 0; k < RA; ++k) v[k] = at[RB * k * PX];
        line_a_inv<T, N>(v, b, tw);
#pragma unroll
        for (int k = 0; k < RA; ++k) at[RB * k * PX] = v[k];
      }
      __syncthreads();
      for (int w = tid; w < PG * RA * N; w += NT) {
        const int l = w % N, t = w / N, ka = t % RA, j = t / RA;
        C* at = buf + (j * N + l) * PX + RB * ka;
        C v[RB];
#pragma unroll
        for (int k = 0; k < RB; ++k) v[k] = at[k];
        Dft<T, RB, true>::run(v);
#pragma unroll
        for (int k = 0; k < RB; ++k) at[k] = v[k];
      }
      __syncthreads();
      for (int w = tid; w < PG * RB * N; w += NT) {
        const int l = w % N, t = w / N, b = t % RB, j = t / RB;
        C* at = buf + (j * N + l) * PX + b;
        C v[RA];
#pragma unroll
        for (int k = 0; k < RA; ++k) v[k] = at[RB * k];
        line_a_inv<T, N>(v, b, tw);
#pragma unroll
        for (int k = 0; k < RA; ++k) at[RB * k] = v[k];
      }
      __syncthreads();
#pragma unroll 1
      for (int i = tid; i < NN; i += NT) {
        const int y = i / N, x = i - y * N;
#pragma unroll
        for (int j = 0; j < PG; ++j) {
          const C wv = buf[(j * N + y) * PX + x];
          T sw[2];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int sl = 2 * j + h, c = sl % 3, z = zg + sl / 3;
            sw[h] = T(0);
            if (z >= ZC) continue;
            sw[h] = __ldg(sc + size_t(c) * NV + z * NN + i) * (h ? wv.y : wv.x);
            ms[c] += double(sw[h]);
            if (z == 0) {
              if (TX) store_async(down_sw + unsigned((c * NN + i) * sizeof(T)), sw[h], down_tx);
              else hsw[size_t(rank) * PL + c * NN + i] = sw[h];
            }
            if (!Cfg::SWS) swg[(z * 3 + c) * NN + i] = sw[h];
          }
          if (Cfg::SWS) buf[(j * N + y) * PX + x] = cmk<C>(sw[0], sw[1]);
        }
      }
    }
    cluster_publish<Cfg, 3, TX>(ms, wsum, slot1, rank, bar, phase, &bar->tx[1], unsigned(PL * sizeof(T)));
    cluster_collect<Cfg, 3, TX>(ms, slot1, bar, phase, &bar->tx[1], tphase1);
    // -------------------------------------------------------------------------- direction
    {
      const T m[3] = {T(ms[0] / double(NV)), T(ms[1] / double(NV)), T(ms[2] / double(NV))};
      const T beta = T(beta64);
      const T* top = hsw + size_t(up) * PL;
#pragma unroll 1
      for (int i = tid; i < NN; i += NT) {
        const int y = i / N, x = i - y * N;
#pragma unroll
        for (int sl = 0; sl < SL; ++sl) {
          const int c = sl % 3, z = sl / 3;
          T v;
          if (Cfg::SWS) {
            const C wv = buf[((sl / 2) * N + y) * PX + x];
            v = sl % 2 ? wv.y : wv.x;
          } else {
            v = swg[(z * 3 + c) * NN + i];
          }
          v -= m[c];
          T* o = p_own + z * PL + 3 * i + c;
          *o = first ? v : v + beta * *o;
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const T v = (TX ? sw_in[c * NN + i] : __ldcg(top + c * NN + i)) - m[c];
          T* o = p_top + 3 * i + c;
          *o = first ? v : v + beta * *o;
        }
      }
    }
    __syncthreads();
    if (*(volatile int*)&bar->dead) break;
    first = false;
    plain = false;
  }
  // No block leaves while another may still reach into its shared memory. A dead block reports and
  // stays until every other one has given up too (they wait at most kClusterWaitClocks each).
  cluster_sync_all<CL>(bar, phase);
  if (*(volatile int*)&bar->dead) {
    if (tid == 0) atomicExch(A.counters + 2, 1);
    for (const long long t0 = clock64(); clock64() - t0 < 4 * kClusterWaitClocks;) {}
    return;
  }
  // x += d; the record the certification and the restart decision read
  double* x = A.x + off;
  for (int i = tid; i < ZC * NN; i += NT) {
    const int z = i / NN, e = i - z * NN;
#pragma unroll
    for (int c = 0; c < 3; ++c) x[3 * size_t(i) + c] += double(d[(z * 3 + c) * NN + e]);
  }
  if (rank == 0 && tid == 0) {
    O.iterations = it;
    O.bad = bad;
    if (sizeof(T) == 4) {
      O.touched += reps;
      atomicMax(A.counters + 3, O.touched);
    }
  }
}

// The kernel of a grid and precision, with its launch shape.
struct ResidentKernel {
  const void* fn;
  int n, prec, cl, nt;
  size_t smem, halo;
};

template <class Cfg> ResidentKernel resident_entry() {
  ResidentKernel k;
  k.fn = reinterpret_cast<const void*>(&k_resident_pcg<Cfg>);
  k.n = Cfg::N;
  k.prec = sizeof(typename Cfg::T) == 4 ? PGJ_FP32 : PGJ_FP64;
  k.cl = Cfg::CL;
  k.nt = Cfg::NT;
  k.smem = Cfg::smem;
  k.halo = Cfg::halo;
  return k;
}

}  // namespace pgj
