// Tile geometry and the packed checkerboard half-sweep of the 3D polynomial solves
// (cn3d_poly.cu: a whole step; cn3d.cu: the periodic preconditioner).
#pragma once

#include <cuda_runtime.h>

#include "tp_common.cuh"

namespace tp {

constexpr int kPW = 64, kPR = 8, kPWarps = 8, kPH = kPR * kPWarps;  // tile width, rows per warp, warps, tile height
constexpr int kPThreads = 32 * kPWarps;
constexpr int kPolyMaxDeg = 10, kPolyMaxHalo = 16;

// Two complex64 values of adjacent columns, each a packed register pair: sums and
// real weights run as packed fp32 operations (one issue slot for both parts).
struct cpair {
  unsigned long long a, b;
};
__device__ __forceinline__ unsigned long long pk(float x, float y) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 upk(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ cpair to_pair(float4 v) { return {pk(v.x, v.y), pk(v.z, v.w)}; }
__device__ __forceinline__ float4 to_f4(cpair v) {
  const float2 a = upk(v.a), b = upk(v.b);
  return make_float4(a.x, a.y, b.x, b.y);
}

// The real weights of a thread's neighbours, each in both halves of a pair:
// left and right of its two columns, and the interior row weight.
struct PolyWeights {
  unsigned long long l0, r0, l1, r1, row;
};

// Weighted neighbour sums of both columns of one row: S = sum of real weights
// times neighbours (the couplings are i times the weights), in the order of
// cn3d.cu's stencils, so that a right-hand side from either is the same to the
// bit: u + d then rounds alike on both marches, and results differ by the solves
// alone.  EDGE: rw holds the row's own weights {previous row, next row, columns}.
template <bool EDGE>
__device__ __forceinline__ cpair poly_sum(const cpair &cur, const cpair &prev, const cpair &next, const PolyWeights &w,
                                          const float4 *rw) {
  const float2 lo = upk(cur.a), hi = upk(cur.b);
  const unsigned long long west = pk(__shfl_up_sync(0xffffffffu, hi.x, 1), __shfl_up_sync(0xffffffffu, hi.y, 1));
  const unsigned long long east = pk(__shfl_down_sync(0xffffffffu, lo.x, 1), __shfl_down_sync(0xffffffffu, lo.y, 1));
  cpair s;
  s.a = fma2(w.r0, cur.b, mul2(w.l0, west));
  s.b = fma2(w.r1, east, mul2(w.l1, cur.a));
  if (EDGE) {
    const float4 v = *rw;
    const unsigned long long x = pk(v.x, v.x), y = pk(v.y, v.y), z = pk(v.z, v.z);
    s.a = fma2(y, next.a, fma2(x, prev.a, mul2(z, s.a)));
    s.b = fma2(y, next.b, fma2(x, prev.b, mul2(z, s.b)));
  } else {
    s.a = fma2(w.row, next.a, fma2(w.row, prev.a, s.a));
    s.b = fma2(w.row, next.b, fma2(w.row, prev.b, s.b));
  }
  return s;
}
// The same for one pixel of colour C in row I of the thread's strip (rows start
// even): colour A (0) is column 0 in even rows and column 1 in odd ones.  o, prev
// and next are the other colour's pixels in this row and its neighbours.
template <bool EDGE, int COL>
__device__ __forceinline__ unsigned long long poly_half(unsigned long long o, unsigned long long prev,
                                                        unsigned long long next, const PolyWeights &w,
                                                        const float4 *rw) {
  const float2 v = upk(o);
  const unsigned long long side = COL == 0 ? pk(__shfl_up_sync(0xffffffffu, v.x, 1), __shfl_up_sync(0xffffffffu, v.y, 1))
                                           : pk(__shfl_down_sync(0xffffffffu, v.x, 1),
                                                __shfl_down_sync(0xffffffffu, v.y, 1));
  unsigned long long s = COL == 0 ? fma2(w.l0, side, mul2(w.r0, o)) : fma2(w.l1, o, mul2(w.r1, side));
  if (EDGE) {
    const float4 r = *rw;
    s = fma2(pk(r.z, r.z), s, fma2(pk(r.x, r.x), prev, mul2(pk(r.y, r.y), next)));
  } else {
    s = fma2(w.row, add2(prev, next), s);
  }
  return s;
}
// c + j s (complex)
__device__ __forceinline__ unsigned long long cmadd(float jx, float jy, unsigned long long s, unsigned long long c) {
  const float2 sv = upk(s), cv = upk(c);
  return pk(fmaf(jx, sv.x, fmaf(-jy, sv.y, cv.x)), fmaf(jx, sv.y, fmaf(jy, sv.x, cv.y)));
}

}  // namespace tp
