// A displacement (or force) triple and its packed FP32 form, shared by the element kernels.
#pragma once
#include "pgj_common.cuh"

namespace pgj {

// Three displacement components of one node or mode. FP32 keeps (x, y) as one packed pair, so an
// add or subtract of two triples is two instructions on sm_100 instead of three. A packed add
// rounds like a scalar one, but the compiler no longer fuses a preceding product into it (as it
// does in scalar code), so FP32 results differ from a scalar build in the last bits.
template <typename T>
struct Tri {
  T x, y, z;
  __device__ __forceinline__ T get(int c) const { return c == 0 ? x : (c == 1 ? y : z); }
  static __device__ __forceinline__ Tri make(T a, T b, T c) { return Tri{a, b, c}; }
  static __device__ __forceinline__ Tri load(const T* p) { return Tri{p[0], p[1], p[2]}; }
  __device__ __forceinline__ void store(T* p) const { p[0] = x; p[1] = y; p[2] = z; }
  friend __device__ __forceinline__ Tri operator+(Tri a, Tri b) { return Tri{a.x + b.x, a.y + b.y, a.z + b.z}; }
  friend __device__ __forceinline__ Tri operator-(Tri a, Tri b) { return Tri{a.x - b.x, a.y - b.y, a.z - b.z}; }
};
template <>
struct Tri<float> {
  float2 xy;
  float z;
  __device__ __forceinline__ float get(int c) const { return c == 0 ? xy.x : (c == 1 ? xy.y : z); }
  static __device__ __forceinline__ Tri make(float a, float b, float c) { return Tri{make_float2(a, b), c}; }
  static __device__ __forceinline__ Tri load(const float* p) { return Tri{make_float2(p[0], p[1]), p[2]}; }
  __device__ __forceinline__ void store(float* p) const { p[0] = xy.x; p[1] = xy.y; p[2] = z; }
  friend __device__ __forceinline__ Tri operator+(Tri a, Tri b) { return Tri{__fadd2_rn(a.xy, b.xy), a.z + b.z}; }
  friend __device__ __forceinline__ Tri operator-(Tri a, Tri b) {
    return Tri{__fadd2_rn(a.xy, make_float2(-b.xy.x, -b.xy.y)), a.z - b.z};
  }
};

}  // namespace pgj
