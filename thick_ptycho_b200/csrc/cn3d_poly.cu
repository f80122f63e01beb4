// 3D Crank-Nicolson march with each slice solved by a fixed polynomial of its
// scaled off-diagonal part, one kernel per step.
//
// A step solves (I - P_s) d = b, P_s = sigma*T(K + diag c_s), b = (P_r + P_s) u
// + src, u_new = u + d (the delta form of cn3d.cu).  With D = I - diag(P_s) and
// J = D^{-1} offdiag(P_s) the system is (I - J) d = D^{-1} b = g.  The off-
// diagonals of K are purely imaginary (mu = i dz / (4 k dx^2)), so the spectrum
// of J lies close to a segment [-i tau, i tau] of the imaginary axis with
// tau = max row sum of |J|, and the Chebyshev residual polynomial of that
// segment gives d = p_m(J) g, p_m(z) = (1 - q_m(z)) / (1 - z), q_m(z) =
// T_m(z / (i tau)) / T_m(1 / (i tau)): the error falls by ~(tau / 2)^m.  At the
// paraxial sampling this path is used at (tau ~ 0.08 at wavelength 0.5 with
// unit steps) m = 6 reaches 2e-8, against ~1.15 FFT-preconditioned BiCGStab
// iterations per solve: 11 kernels and 34 passes over the probes' vectors per
// step become one kernel that reads u once and writes it once.
//
// The 5-point stencil couples only pixels of opposite colour (checkerboard), so
// the Horner recurrence y <- a_k g + J y needs one colour per power of J: y_k
// lives on colour A for odd k and B for even k, ends in d on colour B, and the
// other half of the solution is one exact substitution d^A = g^A + (J d)^A.  A
// solve of even degree m costs m half-sweeps, and only colour B has a residual.
//
// One CTA owns a tile of 64 x 64 pixels (8 warps of 8 rows, two adjacent columns
// per lane: one pixel of each colour) of one image for a group of probes;
// D^{-1} of its 16 pixels stays in a thread's registers for all of them, and so
// do g and y, whose neighbours come from the lane's own registers (the other
// column, the rows above and below), one warp shuffle (left or right) and, at
// the warp's first and last row, shared memory.  A tile computes a core smaller
// than itself: the value of a pixel at the core's edge depends on what is h rows
// outside it only through |J|^h, so a halo of h = 1 + log(1e-8) / log(max |J_ij|) pixels
// (6 at mu = 0.02 and |D| ~ 1) gives the core to below complex64 round-off, whatever m.
// The tiles of u arrive by tiled tensor copies (zero outside the image),
// double-buffered over the group's probes.  Each solve is judged by its true
// residual, as in the Krylov march, but tile by tile with the tile's own d in its halo:
// what the halo leaves out does not show in it.
//
// 256 x 256, 64 probes, m = 6: a forward step to the exit 45.4 us, keeping the field
// 47.6, an exact adjoint step with the gradient 58.6; both marches over 255 slices 191 ->
// 27.4 ms against the Krylov march with transforms (90 x 75 x 48, 9 probes, forward: 6.5 ->
// 0.37 ms).  The schedulers issue in 52 % of a step's cycles and DRAM is 11 % busy; a warp
// waits for the fixed latency of its own arithmetic, for shared memory and shuffles and at
// the exchanges' barriers, about one issue's time each, with 16 warps per SM to cover it.
// Four rows per warp and 12, 14 or 16 warps per CTA (80, 72, 64 registers) were slower
// (55.8, 57.4 and 53.8 us against 42.7 with fp32 norms): twice the exchanges, and taller
// halos where the tile shrinks.
#include <cuda.h>
#include <math.h>
#include <string.h>

#include <complex>
#include <mutex>
#include <type_traits>

#include "cn3d_poly.cuh"
#include "cn3d_poly_dev.cuh"
#include "tp_errors.h"
#include "tpcuda.h"

#ifndef TP_C128_CHECK
namespace tp {

namespace {

struct PolyCheck {
  // bits of the largest row and column sums of |J|, the largest |arg D| and the largest
  // 1 / |D| (non-negative floats)
  unsigned tau, tau_col, arg, inv;
  int bad;
};

struct PolySlices {
  const void *field;
  int nf, nb, N, nz, L, dtype, is_delta, exact, conj_t;
  double sigma, k, dz;
  const float2 *kc, *kw, *ke, *ks, *kn;
  const float2 *colw;
  const float4 *roww;
  float my;  // the row coupling away from the first and last two rows
};

__device__ __forceinline__ double2 poly_coef(const PolySlices &q, size_t idx) {
  double2 v;
  if (q.dtype == TP_C128) {
    v = static_cast<const double2 *>(q.field)[idx];
  } else {
    const float2 w = static_cast<const float2 *>(q.field)[idx];
    v = z2(w.x, w.y);
  }
  const double2 d = q.is_delta ? v : z2(v.x - 1.0, v.y);
  if (!q.exact) return z2(q.k * d.y, -q.k * d.x);
  const double2 w = zadd(zscale(d, 2.0), zmul(d, d));
  return z2(0.5 * q.k * w.y, -0.5 * q.k * w.x);
}

// Column weights {west, east} and row weights {south, north, x factor}: the
// imaginary couplings of sigma*T(K) as products of one-dimensional factors.
__global__ void c3_poly_weights_kernel(const PolySlices q, float2 *colw, float4 *roww) {
  const int br = q.nb / 2, fr = q.nf / 2;
  for (int f = threadIdx.x; f < q.nf; f += blockDim.x) {
    const int i = br * q.nf + f;
    colw[f] = make_float2(f > 0 ? q.kw[i].y : 0.f, f + 1 < q.nf ? q.ke[i].y : 0.f);
  }
  const float2 w0 = q.kw[br * q.nf + fr];
  for (int b = threadIdx.x; b < q.nb; b += blockDim.x) {
    const int i = b * q.nf + fr;
    const float2 w = q.kw[i];
    roww[b] = make_float4(b > 0 ? q.ks[i].y : 0.f, b + 1 < q.nb ? q.kn[i].y : 0.f,
                          (w.x == w0.x && w.y == w0.y) ? 1.f : 0.f, 0.f);
  }
}

// Diagonals of slices s_lo .. s_hi (slice-major, from the node-major index
// field, through a transposing tile), and over every slice of the call's range
// the bounds of J; rows 0 of the grid also compare K's couplings with the
// products of the weights.  Grid (ceil(N / 32), ceil(slices / 32)), block (32, 8).
__global__ void __launch_bounds__(256) c3_poly_slices_kernel(const PolySlices q, int s_first, int s_last, int s_lo,
                                                             int s_hi, float2 *cd, PolyCheck *chk) {
  __shared__ float2 tile[32][33];
  const int i0 = blockIdx.x * 32, s0 = s_first + blockIdx.y * 32;
  float tau = 0.f, tcol = 0.f, arg = 0.f, inv = 0.f;
  int bad = 0;
  for (int r = threadIdx.y; r < 32; r += 8) {
    const int i = i0 + r, s = s0 + threadIdx.x;
    if (i >= q.N || s > s_last) continue;
    const size_t base = (size_t)i * q.nz;
    const double2 c = zscale(zadd(poly_coef(q, base + s - 1), poly_coef(q, base + s)), 0.25 * q.dz);
    const double2 v = zscale(q.conj_t ? zconj(c) : c, q.sigma);
    const float2 kc = q.kc[i];
    const float2 d = make_float2((float)(kc.x + v.x), (float)(kc.y + v.y));
    tile[r][threadIdx.x] = d;
    if (chk != nullptr) {
      const int f = i % q.nf, b = i / q.nf;
      const float2 cw = q.colw[f];
      const float4 rw = q.roww[b];
      const float sum = (fabsf(cw.x) + fabsf(cw.y)) * rw.z + fabsf(rw.x) + fabsf(rw.y);
      if (sum > 0.f) {
        const float dr = 1.f - d.x, di = -d.y;
        const float n = sqrtf(dr * dr + di * di), t = sum / n;
        if (!(t < 1e6f && n < 1e12f)) bad = 1;  // (an infinite D would pass as t = 0)
        tau = fmaxf(tau, t);
        inv = fmaxf(inv, 1.f / n);
        // what row i's element reaches: its neighbours' couplings back to it
        const float col = ((f + 1 < q.nf ? fabsf(q.colw[f + 1].x) : 0.f) + (f > 0 ? fabsf(q.colw[f - 1].y) : 0.f)) * rw.z +
                          (b + 1 < q.nb ? fabsf(q.roww[b + 1].x) : 0.f) + (b > 0 ? fabsf(q.roww[b - 1].y) : 0.f);
        tcol = fmaxf(tcol, col / n);
        arg = fmaxf(arg, fabsf(atan2f(di, dr)));
      } else {
        const float dr = 1.f - d.x, n2 = dr * dr + d.y * d.y;
        if (!(n2 > 1e-6f && n2 < 1e12f)) bad = 1;
      }
      if (blockIdx.y == 0 && threadIdx.x == 0) {
        auto differs = [](float2 v2, float im) { return v2.x != 0.f || v2.y != im; };
        if ((f > 0 && differs(q.kw[i], cw.x * rw.z)) || (f + 1 < q.nf && differs(q.ke[i], cw.y * rw.z)) ||
            (b > 0 && differs(q.ks[i], rw.x)) || (b + 1 < q.nb && differs(q.kn[i], rw.y)))
          bad = 1;
        if (b > 1 && b < q.nb - 2 && (rw.x != q.my || rw.y != q.my || rw.z != 1.f)) bad = 1;
      }
    }
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += 8) {
    const int s = s0 + r, i = i0 + threadIdx.x;
    if (i < q.N && s >= s_lo && s <= s_hi) cd[(size_t)(s - s_lo) * q.N + i] = tile[threadIdx.x][r];
  }
  if (chk == nullptr) return;
  for (int o = 16; o > 0; o >>= 1) {
    tau = fmaxf(tau, __shfl_down_sync(0xffffffffu, tau, o));
    tcol = fmaxf(tcol, __shfl_down_sync(0xffffffffu, tcol, o));
    arg = fmaxf(arg, __shfl_down_sync(0xffffffffu, arg, o));
    inv = fmaxf(inv, __shfl_down_sync(0xffffffffu, inv, o));
    bad |= __shfl_down_sync(0xffffffffu, bad, o);
  }
  if (threadIdx.x == 0) {
    // most blocks do not raise the maxima: read before the atomic
    const volatile PolyCheck *c = chk;
    if (__float_as_uint(tau) > c->tau) atomicMax(&chk->tau, __float_as_uint(tau));
    if (__float_as_uint(tcol) > c->tau_col) atomicMax(&chk->tau_col, __float_as_uint(tcol));
    if (__float_as_uint(arg) > c->arg) atomicMax(&chk->arg, __float_as_uint(arg));
    if (__float_as_uint(inv) > c->inv) atomicMax(&chk->inv, __float_as_uint(inv));
    if (bad) atomicOr(&chk->bad, 1);
  }
}

struct PolyStep {
  int nf, nb, N, P, G;
  int tiles_x, hx, hy, cw, ch;
  int m;
  float a[kPolyMaxDeg];
  float my;  // interior row coupling
  const float2 *cdl, *cdr;
  const float2 *colw;
  const float4 *roww;
  const float2 *u;
  float2 *un;
  int sel;    // which state vector u is (tensor map coordinate)
  int use_u;  // 0: the first step of the exact adjoint (zero state, source only)
  const float2 *src_exit, *src_shared;
  float2 *store;         // the step's slice of u_store, probe stride store_stride
  float keep;            // what is stored: u_new + keep u (keep = 1: pair sums)
  size_t store_stride;
  double2 *norms;  // per probe: ||b||^2, ||b - (I - P) d||^2
  // gradient (exact adjoint): the slice's accumulator += sum_p u_new conj(f1 + f0),
  // f1 and f0 the forward field at the slice's two nodes (probe stride
  // store_stride; f0 NULL: f1 is their sum)
  const float2 *f0, *f1;
  float2 *grad;
};

struct PolySmem {
  float4 u[2][kPH][kPW / 2];
  float4 dsum[kPH][kPW / 2];
  unsigned long long edge[2][kPWarps - 1][2][kPW / 2];  // row exchange between warps w and w + 1: w's last row, (w + 1)'s first
  float4 roww[kPH];
  double2 red[kPWarps];
  uint64_t bar[2];
};

// One tile and probe group.  EDGE: the tile holds one of the image's first or
// last two rows, whose row couplings may differ from the interior's.
template <bool ALIGNED, bool SRC, int GRAD, bool EDGE>
__device__ __forceinline__ void poly_tile(const CUtensorMap &map, const PolyStep &q, PolySmem &sm, int *err) {
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const int tx = blockIdx.x % q.tiles_x, ty = blockIdx.x / q.tiles_x;
  const int f0 = tx * q.cw - q.hx, b0 = ty * q.ch - q.hy;
  const int gf = f0 + 2 * lane, gb0 = b0 + wp * kPR;
  const int p0 = blockIdx.y * q.G, np = min(q.G, q.P - p0);
  const bool in0 = gf >= 0 && gf < q.nf, in1 = gf + 1 >= 0 && gf + 1 < q.nf;
  const bool staged = ALIGNED && (!SRC || q.use_u);
  constexpr uint32_t kTile = kPH * kPW * sizeof(float2);
  if (ALIGNED && threadIdx.x == 0) {
    mbar_init(&sm.bar[0], 1);
    mbar_init(&sm.bar[1], 1);
    fence_mbar_init();
  }
  __syncthreads();
  auto issue = [&](int j) {  // thread 0: probe j's tile of u
    const int buf = GRAD == 2 ? 0 : j & 1;
    mbar_arrive_expect_tx(&sm.bar[buf], kTile);
    tma_load_4d(sm.u[buf], &map, f0, b0, p0 + j, q.sel, &sm.bar[buf]);
  };
  // The next step's CTAs may start as this one's leave: what they do before
  // their own wait reads only the slices' diagonals and the weights.
  pdl_trigger();
  // weights and diagonals of this thread's pixels; zero outside the image, so
  // that g and y stay zero there
  float2 cw0 = make_float2(0.f, 0.f), cw1 = cw0;
  if (in0) cw0 = q.colw[gf];
  if (in1) cw1 = q.colw[gf + 1];
  if (lane == 0) cw0.x = 0.f;
  if (lane == 31) cw1.y = 0.f;
  for (int r = threadIdx.x; r < kPH; r += kPThreads) {
    const int b = b0 + r;
    sm.roww[r] = (b >= 0 && b < q.nb) ? q.roww[b] : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  const PolyWeights w = {pk(cw0.x, cw0.x), pk(cw0.y, cw0.y), pk(cw1.x, cw1.x), pk(cw1.y, cw1.y), pk(q.my, q.my)};
  // every load before the first use, outside pixels from a clamped address
  float4 Ji[kPR], Dr[kPR];  // i D^{-1} of the two columns
#pragma unroll
  for (int i = 0; i < kPR; ++i) {
    const int row = min(max(gb0 + i, 0), q.nb - 1) * q.nf;
    if (ALIGNED) {
      const int at = row + min(max(gf, 0), q.nf - 2);
      Ji[i] = *reinterpret_cast<const float4 *>(q.cdl + at);
      Dr[i] = *reinterpret_cast<const float4 *>(q.cdr + at);
    } else {
      const int c0 = row + min(max(gf, 0), q.nf - 1), c1 = row + min(max(gf + 1, 0), q.nf - 1);
      const float2 l0 = q.cdl[c0], l1 = q.cdl[c1], r0 = q.cdr[c0], r1 = q.cdr[c1];
      Ji[i] = make_float4(l0.x, l0.y, l1.x, l1.y);
      Dr[i] = make_float4(r0.x, r0.y, r1.x, r1.y);
    }
  }
#pragma unroll
  for (int i = 0; i < kPR; ++i) {
    const int b = gb0 + i;
    const bool row = b >= 0 && b < q.nb;
    float4 dl = Ji[i], dr = Dr[i];
    if (!row || !in0) dl.x = dl.y = dr.x = dr.y = 0.f;
    if (!row || !in1) dl.z = dl.w = dr.z = dr.w = 0.f;
    sm.dsum[wp * kPR + i][lane] = make_float4(dl.x + dr.x, dl.y + dr.y, dl.z + dr.z, dl.w + dr.w);
    // i / (1 - d) = (di + i dr) / |1 - d|^2 with 1 - d = dr - i (-di)
    const float ax = 1.f - dl.x, ay = -dl.y, az = 1.f - dl.z, aw = -dl.w;
    const float na = 1.f / fmaf(ax, ax, ay * ay), nz = 1.f / fmaf(az, az, aw * aw);
    Ji[i].x = (row && in0) ? ay * na : 0.f;
    Ji[i].y = (row && in0) ? ax * na : 0.f;
    Ji[i].z = (row && in1) ? aw * nz : 0.f;
    Ji[i].w = (row && in1) ? az * nz : 0.f;
  }
  pdl_wait();  // the step before is complete
  __syncthreads();
  if (staged && threadIdx.x == 0) {
    issue(0);
    if (GRAD != 2 && np > 1) issue(1);
  }
  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
  const bool core0 = 2 * lane >= q.hx && 2 * lane < q.hx + q.cw && in0;
  // this warp's rows in the core (a bit each), and the thread's first pixel
  unsigned rows = 0;
#pragma unroll
  for (int i = 0; i < kPR; ++i) {
    const int r = wp * kPR + i;
    if (r >= q.hy && r < q.hy + q.ch && b0 + r < q.nb) rows |= 1u << i;
  }
  const int at0 = gb0 * q.nf + gf;
  const bool core1 = 2 * lane + 1 >= q.hx && 2 * lane + 1 < q.hx + q.cw && in1;
  for (int j = 0; j < np; ++j) {
    const int p = p0 + j, buf = (ALIGNED && GRAD != 2) ? (j & 1) : 0;
    const ptrdiff_t fo0 = (ptrdiff_t)p * (ptrdiff_t)q.store_stride + at0;
    if (GRAD == 2) {
      // the forward pair sums of this thread's own pixels, on their way while the
      // slice is solved (no tensor copy: those of u would queue behind its misses)
#pragma unroll
      for (int i = 0; i < kPR; ++i)
        if (core0 && ((rows >> i) & 1u)) cp_async16(&sm.u[1][wp * kPR + i][lane], q.f1 + fo0 + i * q.nf);
    }
    if (staged) {
      const uint32_t phase = (uint32_t)((GRAD == 2 ? j : j >> 1) & 1);
      const bool got = mbar_wait_bounded(&sm.bar[buf], phase, err);
      if (__syncthreads_or(!got)) {
        // give up: the copies in flight land before the CTA exits
        cp_async_wait_all();
        if (threadIdx.x == 0) {
          mbar_wait_bounded(&sm.bar[buf], phase, nullptr);
          if (GRAD != 2 && j + 1 < np) mbar_wait_bounded(&sm.bar[buf ^ 1], (uint32_t)(((j + 1) >> 1) & 1), nullptr);
        }
        __syncthreads();
        return;
      }
    } else {
#pragma unroll
      for (int i = 0; i < kPR; ++i) {
        const int b = gb0 + i;
        float4 v = zero4;
        if (q.use_u && b >= 0 && b < q.nb) {
          const float2 *src = q.u + (size_t)p * q.N + (size_t)b * q.nf + gf;
          if (in0) v.x = src[0].x, v.y = src[0].y;
          if (in1) v.z = src[1].x, v.w = src[1].y;
        }
        sm.u[buf][wp * kPR + i][lane] = v;
      }
      __syncthreads();
    }
    if (GRAD == 1 && ALIGNED) {
      // the forward field's rows on their way into L2 while the slice is solved
      const int i = lane >> 1, b = gb0 + i, r = wp * kPR + i;
      if (lane < 2 * kPR && ((lane & 1) || q.f0 != nullptr) && r >= q.hy && r < q.hy + q.ch && b < q.nb) {
        const int c0 = f0 + q.hx, cols = min(q.cw, q.nf - c0);
        const float2 *src = ((lane & 1) ? q.f1 : q.f0) + (size_t)p * q.store_stride + (size_t)b * q.nf + c0;
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(cols * (int)sizeof(float2)) : "memory");
      }
    }
    const float4(*ut)[kPW / 2] = sm.u[buf];
    const cpair zero2 = {0ull, 0ull};
    cpair g[kPR];
    unsigned long long ya[kPR], yb[kPR];  // the newest y of colours A and B
    // ||b||^2 and ||b - (I - P) d||^2, fp64 sums as the Krylov march's (256 x 256, 64
    // probes: 42.9 -> 45.4 us per step; with branches in the place of the selects 50.7)
    double nb2 = 0.0, nr2 = 0.0;
    // g = D^{-1} (dsum u + 2 K_off u + src), y_{m-1} = a_{m-1} g on colour A
    {
      const unsigned long long am = pk(q.a[q.m - 1], q.a[q.m - 1]);
      cpair prev = wp > 0 ? to_pair(ut[wp * kPR - 1][lane]) : zero2, cur = to_pair(ut[wp * kPR][lane]);
#pragma unroll
      for (int i = 0; i < kPR; ++i) {
        const int r = wp * kPR + i, b = gb0 + i;
        const cpair next = r + 1 < kPH ? to_pair(ut[r + 1][lane]) : zero2;
        float4 bv = zero4;
        if (!SRC || q.use_u) {
          const float4 ds = sm.dsum[r][lane], uc = to_f4(cur);
          const float4 s = to_f4(poly_sum<EDGE>(cur, prev, next, w, &sm.roww[r]));
          bv.x = fmaf(ds.x, uc.x, fmaf(-ds.y, uc.y, -2.f * s.y));
          bv.y = fmaf(ds.x, uc.y, fmaf(ds.y, uc.x, 2.f * s.x));
          bv.z = fmaf(ds.z, uc.z, fmaf(-ds.w, uc.w, -2.f * s.w));
          bv.w = fmaf(ds.z, uc.w, fmaf(ds.w, uc.z, 2.f * s.z));
        }
        if (SRC) {
          if (b >= 0 && b < q.nb) {
            const size_t at = (size_t)b * q.nf + gf;
            if (q.src_exit != nullptr) {
              const float2 *src = q.src_exit + (size_t)p * q.N + at;
              if (in0) bv.x += src[0].x, bv.y += src[0].y;
              if (in1) bv.z += src[1].x, bv.w += src[1].y;
            }
            if (q.src_shared != nullptr) {
              const float2 *src = q.src_shared + at;
              if (in0) bv.x += src[0].x, bv.y += src[0].y;
              if (in1) bv.z += src[1].x, bv.w += src[1].y;
            }
          }
        }
        {
          const bool c0 = ((rows >> i) & 1u) && core0, c1 = ((rows >> i) & 1u) && core1;
          const double x0 = c0 ? bv.x : 0.f, y0 = c0 ? bv.y : 0.f, x1 = c1 ? bv.z : 0.f, y1 = c1 ? bv.w : 0.f;
          nb2 = fma(x0, x0, fma(y0, y0, fma(x1, x1, fma(y1, y1, nb2))));
        }
        // D^{-1} = -i Ji = (Ji.y, -Ji.x)
        g[i].a = pk(fmaf(Ji[i].y, bv.x, Ji[i].x * bv.y), fmaf(Ji[i].y, bv.y, -Ji[i].x * bv.x));
        g[i].b = pk(fmaf(Ji[i].w, bv.z, Ji[i].z * bv.w), fmaf(Ji[i].w, bv.w, -Ji[i].z * bv.z));
        ya[i] = mul2(am, (i & 1) ? g[i].b : g[i].a);
        prev = cur;
        cur = next;
      }
    }
    // the other colour's pixels in the rows above and below the warp's strip, which
    // the neighbouring warps publish; buf alternates from one exchange to the next
    auto exchange = [&](const unsigned long long(&v)[kPR], int buf, unsigned long long &above, unsigned long long &below) {
      if (wp > 0) sm.edge[buf][wp - 1][1][lane] = v[0];
      if (wp + 1 < kPWarps) sm.edge[buf][wp][0][lane] = v[kPR - 1];
      __syncthreads();
      above = wp > 0 ? sm.edge[buf][wp - 1][0][lane] : 0ull;
      below = wp + 1 < kPWarps ? sm.edge[buf][wp][1][lane] : 0ull;
    };
    // a g + J v on colour C, v on the other one
    auto half_sweep = [&](auto colour, float a, const unsigned long long(&v)[kPR], unsigned long long(&out)[kPR]) {
      constexpr int C = decltype(colour)::value;
      unsigned long long prev, below;
      exchange(v, C, prev, below);
      const unsigned long long a2 = pk(a, a);
#pragma unroll
      for (int i = 0; i < kPR; ++i) {
        const unsigned long long next = i + 1 < kPR ? v[i + 1] : below;
        const float4 *rw = &sm.roww[wp * kPR + i];
        if ((C + i) % 2 == 0) {
          const unsigned long long s = poly_half<EDGE, 0>(v[i], prev, next, w, rw);
          out[i] = cmadd(Ji[i].x, Ji[i].y, s, mul2(a2, g[i].a));
        } else {
          const unsigned long long s = poly_half<EDGE, 1>(v[i], prev, next, w, rw);
          out[i] = cmadd(Ji[i].z, Ji[i].w, s, mul2(a2, g[i].b));
        }
        prev = v[i];
      }
    };
#pragma unroll 1
    for (int k = q.m - 2; k >= 0; k -= 2) {
      half_sweep(std::integral_constant<int, 1>{}, q.a[k], ya, yb);
      // y_{k-1}; after y_0 = d on colour B, the substitution for colour A
      half_sweep(std::integral_constant<int, 0>{}, k > 0 ? q.a[k - 1] : 1.f, yb, ya);
    }
    // the residual of colour B, b - (I - P) d = D (g + J d - d), and u + d
    {
      unsigned long long prev, below;
      exchange(ya, 1, prev, below);
      float2 *un = q.un + ((ptrdiff_t)p * q.N + at0);
      float2 *store = q.store + ((ptrdiff_t)p * (ptrdiff_t)q.store_stride + at0);
#pragma unroll
      for (int i = 0; i < kPR; ++i) {
        const int r = wp * kPR + i;
        const bool odd = (i & 1) != 0;
        const unsigned long long next = i + 1 < kPR ? ya[i + 1] : below;
        const unsigned long long s = odd ? poly_half<EDGE, 0>(ya[i], prev, next, w, &sm.roww[r])
                                         : poly_half<EDGE, 1>(ya[i], prev, next, w, &sm.roww[r]);
        if ((rows >> i) & 1u) {
          const float4 uo = ut[r][lane];
          const float2 d0 = upk(odd ? yb[i] : ya[i]), d1 = upk(odd ? ya[i] : yb[i]);
          const int row = i * q.nf;
          const float4 v = make_float4(uo.x + d0.x, uo.y + d0.y, uo.z + d1.x, uo.w + d1.y);
          auto put = [&](float2 *dst, float4 v, bool stream) {
            if (ALIGNED) {
              if (core0) {
                if (stream) __stcs(reinterpret_cast<float4 *>(dst), v);
                else *reinterpret_cast<float4 *>(dst) = v;
              }
            } else {
              if (core0) dst[0] = make_float2(v.x, v.y);
              if (core1) dst[1] = make_float2(v.z, v.w);
            }
          };
          put(un + row, v, false);
          if (q.store != nullptr)
            put(store + row,
                make_float4(fmaf(q.keep, uo.x, v.x), fmaf(q.keep, uo.y, v.y), fmaf(q.keep, uo.z, v.z),
                            fmaf(q.keep, uo.w, v.w)),
                true);
          const float jx = odd ? Ji[i].x : Ji[i].z, jy = odd ? Ji[i].y : Ji[i].w;
          const float2 rg = upk(cmadd(jx, jy, s, odd ? g[i].a : g[i].b)), rd = upk(yb[i]);
          const float rx = rg.x - rd.x, ry = rg.y - rd.y;
          if (odd ? core0 : core1)
            nr2 = fma((double)__fdividef(1.f, fmaf(jx, jx, jy * jy)), fma((double)rx, (double)rx, (double)ry * (double)ry), nr2);
        }
        prev = ya[i];
      }
    }
    if (GRAD != 0) {
      // every row's forward field before the first reduction (Ji and g are done with)
      float4 fs[kPR];
      if (GRAD == 2) cp_async_wait_all();
#pragma unroll
      for (int i = 0; i < kPR; ++i) {
        fs[i] = zero4;
        if (!((rows >> i) & 1u)) continue;
        const ptrdiff_t fo = fo0 + i * q.nf;
        if (GRAD == 2) {
          fs[i] = sm.u[1][wp * kPR + i][lane];
        } else if (ALIGNED) {
          if (core0) {
            fs[i] = __ldcs(reinterpret_cast<const float4 *>(q.f1 + fo));
            if (q.f0 != nullptr) {
              const float4 c0 = *reinterpret_cast<const float4 *>(q.f0 + fo);
              fs[i] = make_float4(c0.x + fs[i].x, c0.y + fs[i].y, c0.z + fs[i].z, c0.w + fs[i].w);
            }
          }
        } else {
          if (core0) fs[i].x = q.f1[fo].x, fs[i].y = q.f1[fo].y;
          if (core1) fs[i].z = q.f1[fo + 1].x, fs[i].w = q.f1[fo + 1].y;
          if (q.f0 != nullptr) {
            if (core0) fs[i].x += q.f0[fo].x, fs[i].y += q.f0[fo].y;
            if (core1) fs[i].z += q.f0[fo + 1].x, fs[i].w += q.f0[fo + 1].y;
          }
        }
      }
      float2 *grad = q.grad + at0;
#pragma unroll
      for (int i = 0; i < kPR; ++i) {
        if (!((rows >> i) & 1u)) continue;
        const float4 uo = ut[wp * kPR + i][lane];
        const float2 d0 = upk((i & 1) ? yb[i] : ya[i]), d1 = upk((i & 1) ? ya[i] : yb[i]);
        const float2 g0 = cmulc(make_float2(uo.x + d0.x, uo.y + d0.y), make_float2(fs[i].x, fs[i].y));
        const float2 g1 = cmulc(make_float2(uo.z + d1.x, uo.w + d1.y), make_float2(fs[i].z, fs[i].w));
        float2 *dst = grad + i * q.nf;
        if (ALIGNED) {
          if (core0) red_add_cx2(reinterpret_cast<float4 *>(dst), make_float4(g0.x, g0.y, g1.x, g1.y));
        } else {
          if (core0) red_add_cx(dst, g0);
          if (core1) red_add_cx(dst + 1, g1);
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      nb2 += __shfl_down_sync(0xffffffffu, nb2, o);
      nr2 += __shfl_down_sync(0xffffffffu, nr2, o);
    }
    if (lane == 0) sm.red[wp] = make_double2(nb2, nr2);
    __syncthreads();  // every thread is done with this probe's tile; the partial norms are in
    if (threadIdx.x == 0) {
      if (GRAD == 2) {
        if (staged && j + 1 < np) {
          fence_proxy_async_smem();
          issue(j + 1);
        }
      } else if (staged && j + 2 < np) {
        fence_proxy_async_smem();
        issue(j + 2);
      }
      double sb = 0.0, sr = 0.0;
#pragma unroll
      for (int w = 0; w < kPWarps; ++w) {
        sb += sm.red[w].x;
        sr += sm.red[w].y;
      }
      atomicAdd(&q.norms[p].x, sb);
      atomicAdd(&q.norms[p].y, sr);
    }
  }
}

// SRC: the step has a source, or (use_u = 0) nothing but a source.  GRAD: the step
// adds its gradient contributions (2: from pair sums copied into the place of
// the next probe's u).
template <bool ALIGNED, bool SRC, int GRAD>
__global__ void __launch_bounds__(kPThreads, 2) c3_poly_kernel(const __grid_constant__ CUtensorMap map,
                                                               const __grid_constant__ PolyStep q, int *err) {
  extern __shared__ __align__(128) unsigned char raw[];
  PolySmem &sm = *reinterpret_cast<PolySmem *>(raw);
  const int b0 = (int)(blockIdx.x / q.tiles_x) * q.ch - q.hy;
  if (b0 <= 1 || b0 + kPH > q.nb - 2) poly_tile<ALIGNED, SRC, GRAD, true>(map, q, sm, err);
  else poly_tile<ALIGNED, SRC, GRAD, false>(map, q, sm, err);
}

// Statistics of every solve of the march: m iterations each (none where the
// right-hand side was zero), failures by the true residual.
__global__ void c3_poly_stats_kernel(const double2 *norms, int count, int m, double tol2, int *stats) {
  int iters = 0, failed = 0;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < count; e += gridDim.x * blockDim.x) {
    const double2 v = norms[e];
    if (v.x == 0.0) continue;
    iters += m;
    if (!(v.y <= 100.0 * tol2 * v.x)) ++failed;  // 10x the tolerance, as the Krylov march
  }
  if (iters > 0) {
    atomicAdd(&stats[0], iters);
    atomicMax(&stats[3], m);
  }
  if (failed > 0) atomicAdd(&stats[2], failed);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    atomicAdd(&stats[1], count);
    stats[4] = 2;
  }
}

// u_store's slice of the initial state.
__global__ void c3_poly_first_kernel(int N, int P, const float2 *__restrict__ u, float2 *store, size_t stride) {
  const size_t total = (size_t)P * N;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x)
    store[(e / N) * stride + e % N] = u[e];
}

using EncodeTiled = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                 const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiled encoder() {
  static EncodeTiled fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult qr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &qr) == cudaSuccess &&
        qr == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiled>(f);
    (void)cudaGetLastError();
  });
  return fn;
}

// T_m(w) for complex w.
std::complex<double> chebyshev(int m, std::complex<double> w) {
  std::complex<double> t0 = 1.0, t1 = w;
  if (m == 0) return t0;
  for (int j = 1; j < m; ++j) {
    const std::complex<double> t2 = 2.0 * w * t1 - t0;
    t0 = t1;
    t1 = t2;
  }
  return t1;
}

}  // namespace

// The smallest even degree whose residual polynomial stays below `target` on the
// segment [-i tau, i tau] turned by up to `theta`; 0 if none is allowed.  a[k] are
// the coefficients of p_m.
int poly_degree(double tau, double theta, double target, int max_m, float *a) {
  if (!(tau >= 0.0) || tau > 0.7) return 0;
  if (tau < 1e-3) tau = 1e-3;
  const std::complex<double> it(0.0, tau);
  for (int m = 4; m <= max_m; m += 2) {
    const std::complex<double> scale = chebyshev(m, 1.0 / it);
    const double bound = std::abs(chebyshev(m, std::polar(1.0, theta))) / std::abs(scale);
    if (!(bound <= target)) continue;
    // Chebyshev coefficients t_j of T_m
    double t0[kPolyMaxDeg + 1] = {1.0}, t1[kPolyMaxDeg + 1] = {0.0, 1.0};
    for (int n = 1; n < m; ++n) {
      double t2[kPolyMaxDeg + 1] = {0.0};
      for (int j = 0; j <= m; ++j) t2[j] = (j > 0 ? 2.0 * t1[j - 1] : 0.0) - t0[j];
      for (int j = 0; j <= m; ++j) t0[j] = t1[j], t1[j] = t2[j];
    }
    std::complex<double> pw = 1.0, p = 1.0;  // (i tau)^{-j}
    for (int k = 0; k < m; ++k) {
      p -= t1[k] * pw / scale;
      a[k] = (float)p.real();  // T_m has one parity: real
      pw /= it;
    }
    return m;
  }
  return 0;
}

int c3_poly_march(const C3PolyJob &job, cudaStream_t st, int *ran) {
  *ran = 0;
  const int nf = job.nf, nb = job.nb, N = nf * nb, nz = job.nz, L = nz - 1, P = job.P;
  constexpr int kMaxSlices = 32 * 65535;  // of one launch over all slices
  if (nf > kPolyMaxSide || nb > kPolyMaxSide || job.tol < 4e-7 || L > kMaxSlices) return TP_OK;
  const bool adj_exact = job.mode == TP_MODE_ADJOINT_EXACT;
  const size_t norms_bytes = ((size_t)L * P * sizeof(double2) + 255) & ~size_t(255);
  if (job.scratch_bytes < norms_bytes) return TP_OK;
  size_t cap = (job.scratch_bytes - norms_bytes) / ((size_t)N * sizeof(float2));
  if (cap > (size_t)L) cap = L;
  if (cap < 2) return TP_OK;
  double2 *norms = reinterpret_cast<double2 *>(job.scratch);
  float2 *cd = reinterpret_cast<float2 *>(job.scratch + norms_bytes);

  PolySlices sl{};
  sl.field = job.field;
  sl.nf = nf;
  sl.nb = nb;
  sl.N = N;
  sl.nz = nz;
  sl.L = L;
  sl.dtype = job.dtype;
  sl.is_delta = job.is_delta;
  sl.exact = job.exact;
  sl.conj_t = job.conj_t;
  sl.sigma = job.sigma;
  sl.k = job.k;
  sl.dz = job.dz;
  sl.kc = job.kc;
  sl.kw = job.kw;
  sl.ke = job.ke;
  sl.ks = job.ks;
  sl.kn = job.kn;
  sl.colw = job.colw;
  sl.roww = job.roww;
  sl.my = (float)job.mu_y;
  // slices [lo, hi] in cd: all of them, or as many as fit, in the march's order
  const bool backward = job.mode != TP_MODE_FORWARD;
  const int C = (int)cap;
  int lo = backward ? L - C + 1 : 1, hi = backward ? L : C;
  if (lo < 1) lo = 1;
  if (hi > L) hi = L;
  PolyCheck *chk = reinterpret_cast<PolyCheck *>(job.check);
  TP_CHECK_CUDA(cudaMemsetAsync(chk, 0, sizeof(PolyCheck), st));
  c3_poly_weights_kernel<<<1, 512, 0, st>>>(sl, job.colw, job.roww);
  const dim3 sblock(32, 8);
  c3_poly_slices_kernel<<<dim3((N + 31) / 32, (L + 31) / 32), sblock, 0, st>>>(sl, 1, L, lo, hi, cd, chk);
  TP_CHECK_CUDA(cudaGetLastError());
  PolyCheck host{};
  TP_CHECK_CUDA(cudaMemcpyAsync(&host, chk, sizeof(PolyCheck), cudaMemcpyDeviceToHost, st));
  TP_CHECK_CUDA(cudaStreamSynchronize(st));
  if (host.bad) return TP_OK;
  // either norm bounds the spectral radius (a transposed operator's rows are the
  // original's columns: the doubled Neumann couplings add up in one of the two)
  float tau, tcol, theta, inv;
  memcpy(&tau, &host.tau, 4);
  memcpy(&tcol, &host.tau_col, 4);
  if (tcol < tau) tau = tcol;
  memcpy(&theta, &host.arg, 4);
  memcpy(&inv, &host.inv, 4);

  PolyStep q{};
  const double target = 0.1 * (job.tol < 1e-6 ? job.tol : 1e-6);
  q.m = poly_degree(tau, theta, target, kPolyMaxDeg < job.max_iter ? kPolyMaxDeg : job.max_iter, q.a);
  if (q.m == 0) return TP_OK;
  // halo: one pixel for the right-hand side and the reach of 1e-8 of J's largest entry
  // between interior pixels (no more than the polynomial's)
  const double ent = fmax(1e-6, fmax(fabs(job.mu_x), fabs(job.mu_y)) * (double)inv);
  int h = 1 + (ent < 1.0 ? (int)ceil(log(1e-8) / log(ent)) : kPolyMaxHalo);
  if (h > q.m + 1) h = q.m + 1;
  if (h > kPolyMaxHalo) return TP_OK;

  // 16-byte accesses and tensor copies need even rows and aligned outputs
  auto al16 = [](const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  bool aligned = nf % 2 == 0 && al16(job.u_store) && al16(job.exit_out) && al16(job.u_fwd) && al16(job.grad_c) && al16(cd) && al16(job.vec[0]);
  CUtensorMap map{};
  int *err = nullptr;
  if (aligned) {
    EncodeTiled enc = encoder();
    err = device_error_ptr();
    const cuuint64_t dims[4] = {(cuuint64_t)nf, (cuuint64_t)nb, (cuuint64_t)P, 2};
    const cuuint64_t str[3] = {(cuuint64_t)nf * sizeof(float2), (cuuint64_t)N * sizeof(float2), job.vstride};
    const cuuint32_t box[4] = {kPW, kPH, 1, 1}, es[4] = {1, 1, 1, 1};
    aligned = enc != nullptr && err != nullptr &&
              enc(&map, CU_TENSOR_MAP_DATA_TYPE_UINT64, 4, job.vec[0], dims, str, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  }
  q.nf = nf;
  q.nb = nb;
  q.N = N;
  q.P = P;
  q.hx = (h + 1) & ~1;  // tensor copies start at an even column
  q.hy = h;
  q.tiles_x = (nf + kPW - 2 * q.hx - 1) / (kPW - 2 * q.hx);
  const int tiles_y = (nb + kPH - 2 * q.hy - 1) / (kPH - 2 * q.hy);
  q.cw = (((nf + q.tiles_x - 1) / q.tiles_x) + 1) & ~1;
  q.ch = (nb + tiles_y - 1) / tiles_y;
  const int tiles = q.tiles_x * tiles_y;
  int dev = 0, sms = 148;
  TP_CHECK_CUDA(cudaGetDevice(&dev));
  TP_CHECK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  // probes per CTA: as few as give one wave of two CTAs per SM
  const int slots = 2 * sms;
  int groups = slots / tiles;
  if (groups < 1) groups = 1;
  if (groups > P) groups = P;
  q.G = (P + groups - 1) / groups;
  groups = (P + q.G - 1) / q.G;
  q.colw = job.colw;
  q.roww = job.roww;
  q.my = sl.my;
  const size_t smem = sizeof(PolySmem) + 128;
  const int grad = job.grad_c ? (aligned && job.sums ? 2 : 1) : 0;
  using PolyKernel = void (*)(const CUtensorMap, const PolyStep, int *);
  PolyKernel kerns[2];  // without and with a source
  if (aligned && grad == 2) kerns[0] = c3_poly_kernel<true, false, 2>, kerns[1] = c3_poly_kernel<true, true, 2>;
  else if (aligned && grad) kerns[0] = c3_poly_kernel<true, false, 1>, kerns[1] = c3_poly_kernel<true, true, 1>;
  else if (aligned) kerns[0] = c3_poly_kernel<true, false, 0>, kerns[1] = c3_poly_kernel<true, true, 0>;
  else if (grad) kerns[0] = c3_poly_kernel<false, false, 1>, kerns[1] = c3_poly_kernel<false, true, 1>;
  else kerns[0] = c3_poly_kernel<false, false, 0>, kerns[1] = c3_poly_kernel<false, true, 0>;
  for (PolyKernel k : kerns)
    TP_CHECK_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));

  const size_t vec_bytes = (size_t)P * N * sizeof(float2);
  if (job.probes != nullptr)
    TP_CHECK_CUDA(cudaMemcpyAsync(job.vec[0], job.probes, vec_bytes, cudaMemcpyDeviceToDevice, st));
  else
    TP_CHECK_CUDA(cudaMemsetAsync(job.vec[0], 0, vec_bytes, st));
  TP_CHECK_CUDA(cudaMemsetAsync(norms, 0, (size_t)L * P * sizeof(double2), st));
  const bool flip = job.mode == TP_MODE_ADJOINT;
  const size_t stride = (size_t)nz * N;
  if (job.u_store)
    c3_poly_first_kernel<<<296, 256, 0, st>>>(N, P, job.vec[0], job.u_store + (flip ? (size_t)L * N : 0), stride);
  bool fresh = true;
  for (int t = 1; t <= L; ++t) {
    const int s = backward ? L + 1 - t : t;
    const int sr = (adj_exact && t > 1) ? s + 1 : s;
    if (s < lo || s > hi) {  // the next run of slices (with slice s + 1 for the exact adjoint)
      if (backward) {
        hi = sr;
        lo = hi - C + 1 > 1 ? hi - C + 1 : 1;
      } else {
        lo = s;
        hi = lo + C - 1 < L ? lo + C - 1 : L;
      }
      c3_poly_slices_kernel<<<dim3((N + 31) / 32, (hi - lo) / 32 + 1), sblock, 0, st>>>(sl, lo, hi, lo, hi, cd, nullptr);
      fresh = true;
    }
    q.cdl = cd + (size_t)(s - lo) * N;
    q.cdr = cd + (size_t)(sr - lo) * N;
    q.sel = (t - 1) & 1;
    q.u = job.vec[q.sel];
    q.un = (t == L && job.exit_out) ? job.exit_out : job.vec[q.sel ^ 1];
    q.use_u = !(adj_exact && t == 1);
    q.src_exit = t == 1 ? job.src_exit : nullptr;
    q.src_shared = job.src_shared ? job.src_shared + (size_t)(t - 1) * N : nullptr;
    q.store = job.u_store ? job.u_store + (size_t)(flip ? L - t : t) * N : nullptr;
    q.keep = job.sums ? 1.f : 0.f;
    q.store_stride = stride;
    q.norms = norms + (size_t)(t - 1) * P;
    const bool src = q.src_exit != nullptr || q.src_shared != nullptr || !q.use_u;
    if (job.grad_c) {
      q.f0 = job.sums ? nullptr : job.u_fwd + (size_t)(s - 1) * N;
      q.f1 = job.u_fwd + (size_t)s * N;
      q.grad = job.grad_c + (size_t)(s - 1) * N;
    }
    // behind another kernel than a step's: after all of it
    TP_CHECK_CUDA(launch_dependent(kerns[src ? 1 : 0], dim3(tiles, groups), dim3(kPThreads), smem, st, !fresh, map, q, err));
    fresh = false;
  }
  if (job.stats) c3_poly_stats_kernel<<<32, 256, 0, st>>>(norms, L * P, q.m, job.tol * job.tol, job.stats);
  TP_CHECK_CUDA(cudaGetLastError());
  *ran = 1;
  return TP_OK;
}

}  // namespace tp
#endif  // TP_C128_CHECK
