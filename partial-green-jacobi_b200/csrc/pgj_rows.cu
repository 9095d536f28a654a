// Launch of the operator (pgj_rows.cuh): tile choice and instantiations.
#include "pgj_rows.cuh"
#include <algorithm>

namespace pgj {

namespace {
// Threads per block at most. One block of this size, or several smaller ones, fill an SM: the kernel takes about
// 250 registers in FP64 (128 would spill: 2 to 3 times slower) and 150 in FP32, where 256 threads leave latency
// uncovered on large grids (n = 96 93 against 88 us, 128 227 against 205) and 512 spill (n = 64 36 against 27).
constexpr int kThr64 = 256, kThr32 = 384;
// Blocks per SM at most: in FP64 the exchange buffers (49 KB whatever the block's size) leave room for four; in FP32
// for six, and the recurrence's instance has registers for five blocks of two warps.
// Counting eight, as the threads alone would allow, took shapes with a second, nearly empty wave: recurrence operator of
// six loads n = 24 18.5 us FP64, 14.4 mixed (14.3, 12.3 now), n = 30 20.5, 16.4 (14.4, 12.3), n = 32 mixed 15.3 (12.3).
constexpr int kPer64 = 4, kPer32 = 5;

template <typename T, int MODE, typename R, bool COMP, bool VEC>
struct Rows {
  static constexpr bool wide = sizeof(R) == 8;
  static constexpr int THR = wide ? kThr64 : kThr32;
  static constexpr size_t smem = sizeof(R) * 24 * THR + 4 * 32 * 8;
  static constexpr auto fn = k_rows<T, MODE, R, COMP, VEC, THR>;
  static int go(const StencilArgs& A, const StencilGeom& g, int loads, cudaStream_t s) {
    const dim3 grid(g.ntiles, g.nchunks, loads), block(A.n / 2, g.ty + 1);
    fn<<<grid, block, smem, s>>>(A);
    return check_launch();
  }
  static void prepare() { cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)); }
};
}  // namespace

// Tile rows and z chunks for the loads of one design: the shape with the largest share of the chip's threads at
// work on elements that count. Lost are the threads that fill up a warp or an SM, the halo row, rows beyond the
// last tile, the two planes at a chunk's start and end, and the slots of the last wave. Depends on n and the
// loads per design only, so a design's summation order is the same alone and in a batch. Of all shapes
// timed one by one at n = 40, 48, 64, 72 and 96 it is the fastest, but for FP32 at n = 96 (88 against 84 us).
StencilGeom rows_geom(int n, int lpd, bool wide) {
  const int most = wide ? kThr64 : kThr32, nh = n / 2;
  StencilGeom best;
  double top = -1.0;
  for (int ty = 1; ty <= n && nh * (ty + 1) <= most; ++ty) {
    const int tiles = (n + ty - 1) / ty, warps = (nh * (ty + 1) + 31) / 32;
    // blocks per SM: by threads (registers), at most kPer64 or kPer32
    const int per = std::min(most / 32 / warps, wide ? kPer64 : kPer32);
    const double rows = double(n) * nh / (double(tiles) * warps * 32) * double(per * warps * 32) / most;
    for (int nch = 1; nch <= (n / 4 > 1 ? n / 4 : 1); ++nch) {
      const int zc = (n + nch - 1) / nch, chunks = (n + zc - 1) / zc;
      const long slots = 148L * per, blocks = long(lpd) * tiles * chunks, waves = (blocks + slots - 1) / slots;
      const double eff = rows * n / (double(chunks) * (zc + 2)) * double(blocks) / double(waves * slots);
      if (long(tiles) * chunks <= kMaxPartials && eff > top + 1e-9) {
        top = eff;
        best.ty = ty; best.ntiles = tiles; best.zc = zc; best.nchunks = chunks; best.occ = per;
      }
    }
  }
  return best;
}

int launch_stencil(pgj_ctx* c, int mode, int loads, int prec, const void* in, void* out, const double* f,
                   const int32_t* active_ext, cudaStream_t s, const LoadScalars* rel_flags) {
  const bool fp32 = prec == PGJ_FP32;
  // FP32 recurrence operator with FP64 arithmetic (high-contrast mixed solves)
  const bool r64 = fp32 && mode == kPCG && c->op64;
  const StencilGeom& g = fp32 && !r64 ? c->geo32 : c->geo64;
  StencilArgs A = {};
  A.n = c->n; A.ty = g.ty; A.zc = g.zc; A.lpd = c->lpd;
  A.a = c->a; A.in = in; A.out = out; A.f = f; A.active_ext = active_ext;
  A.rel_flags = rel_flags; A.scal = c->scal; A.partials = c->partials; A.kc = c->kc;
  if (mode == kPlain) {
    // a caller's vectors need not be aligned to a pair of values
    const uintptr_t pair = fp32 ? 8 : 16;
    const bool vec = (reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) % pair == 0;
    if (fp32)
      return vec ? Rows<float, kPlain, float, false, true>::go(A, g, loads, s)
                 : Rows<float, kPlain, float, false, false>::go(A, g, loads, s);
    return vec ? Rows<double, kPlain, double, false, true>::go(A, g, loads, s)
               : Rows<double, kPlain, double, false, false>::go(A, g, loads, s);
  }
  if (mode == kResidual)
    return fp32 ? PGJ_ERR_ARGUMENT : Rows<double, kResidual, double, false, true>::go(A, g, loads, s);
  // the plane kernels hold p and q by component
  if (c->four) {
    if (r64) return Rows<float, kPCG, double, true, true>::go(A, g, loads, s);
    return fp32 ? Rows<float, kPCG, float, true, true>::go(A, g, loads, s)
                : Rows<double, kPCG, double, true, true>::go(A, g, loads, s);
  }
  if (r64) return Rows<float, kPCG, double, false, true>::go(A, g, loads, s);
  return fp32 ? Rows<float, kPCG, float, false, true>::go(A, g, loads, s)
              : Rows<double, kPCG, double, false, true>::go(A, g, loads, s);
}

int prepare_rows() {
  Rows<double, kPlain, double, false, true>::prepare();
  Rows<double, kPlain, double, false, false>::prepare();
  Rows<double, kResidual, double, false, true>::prepare();
  Rows<double, kPCG, double, true, true>::prepare();
  Rows<double, kPCG, double, false, true>::prepare();
  Rows<float, kPCG, double, true, true>::prepare();
  Rows<float, kPCG, double, false, true>::prepare();
  Rows<float, kPlain, float, false, true>::prepare();
  Rows<float, kPlain, float, false, false>::prepare();
  Rows<float, kPCG, float, true, true>::prepare();
  Rows<float, kPCG, float, false, true>::prepare();
  return check_launch();
}

}  // namespace pgj
