// 3D angular-spectrum multislice (forward march and its adjoint).
//
// The reference's multislice solver is 2D only (forward_model/multislice/
// ms_solver.py:28-31 rejects a 3D simulation space); this is the same
// propagator on an (n1, n2) transverse grid:
//   psi <- IFFT2(H . FFT2(psi . T_z)),  T_z = exp(i k (n[:, z] - n_medium) dz),
//   H = exp(i (k_z - k) dz),  k_z = sqrt(max(k^2 - k1^2 - k2^2, 0)),
//   k1 = 2 pi fftfreq(n1, d1), k2 = 2 pi fftfreq(n2, d2)
// (the 2D kernel of ms_solver.py:49-72 with the transverse wavenumber made
// two-dimensional).  Element (a, b) of a slice sits at a * n2 + b, the
// C-order flattening of the reference's (nx, ny) arrays.
//
// A 256 x 256 slice (512 KB) does not fit one CTA's shared memory, so each
// slice is two kernels over all probes:
//   rows:    inverse row FFTs of the spectrum W, psi_{z+1} = X_z + result
//            (delta form, X_z = psi_z T_z), store, X_{z+1} = psi_{z+1} T_{z+1},
//            forward row FFTs into W;
//   columns: column FFTs, times (H - 1)/N, inverse column FFTs, in place.
// The field psi and the spectrum W (P x N complex64 each) are updated in place
// by the CTA that owns the rows, so a march needs no ping-pong buffers; at
// 64 probes of 256 x 256 both fit in L2.  T - 1 and H - 1 are kept as
// deviations from one, evaluated in fp64, so the fp32 FFT round-off scales
// with the per-slice update, not the field.
#include <cuda_runtime.h>

#include "fft.cuh"
#include "tp_errors.h"
#include "tpcuda.h"

namespace tp {

constexpr int kMs3Threads = 256;

// host helper of ms2d.cu: the fp64 T - 1 table of an (n_total, nz) index field
int ms_transmission_launch(int n_total, int nz, double k, double dz, double nmr, double nmi, const void *field,
                           int dtype, float2 *trans, cudaStream_t st);

struct Ms3Params {
  int n1, n2, N, nz, L, P;
  const float2 *trans;  // (L, N): T_z - 1
  const float2 *hm1t;   // (H - 1) / N, (n1, n2)
  const float2 *tw1, *tw2;
  float2 *psi;          // (P, N): field (forward) or lambda (adjoint), in place
  float2 *W;            // (P, N): spectrum work buffer, in place
  const float2 *probes, *src_exit, *u_fwd;
  float2 *u_store, *exit_out, *grad_t;
};

enum Ms3Phase : int { kMs3FwdStart = 0, kMs3FwdStep = 1, kMs3BwdStart = 2, kMs3BwdStep = 3 };

// The stages' twiddles of an in-place plan.
__global__ void ms3_twiddle_mix_kernel(const __grid_constant__ MixPlan pl, float2 *tw) {
  mix_twiddles(pl, tw, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

// (H - 1) / N at a * n2 + b, the axes of an in-place plan (stages > 0) by place instead
// of frequency; H - 1 = exp(i th) - 1 = -2 sin^2(th/2) + i sin th.  Less the transforms'
// gain (fft.cuh): `gain` is the share of their constants, those of the twiddles are summed here.
__global__ void ms3_kernel_h_kernel(int n1, int n2, const __grid_constant__ MixPlan p1, const __grid_constant__ MixPlan p2,
                                    const float2 *tw1, const float2 *tw2, double gain, double k, double d1, double d2,
                                    double dz, float2 *hm1t) {
  __shared__ double red[32];
  const int N = n1 * n2, tid = threadIdx.x, nth = blockDim.x;
  gain += cta_sum((p1.stages > 0 ? mix_twiddle_gain(p1, tw1, tid, nth) : four_twiddle_gain(n1, tw1, tid, nth)) +
                        (p2.stages > 0 ? mix_twiddle_gain(p2, tw2, tid, nth) : four_twiddle_gain(n2, tw2, tid, nth)), red);
  const double inv = 1.0 / ((double)N * (1.0 + gain));
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < N; e += gridDim.x * blockDim.x) {
    int a = e / n2, b = e % n2;
    if (p1.stages > 0) a = mix_frequency(p1, a);
    if (p2.stages > 0) b = mix_frequency(p2, b);
    const int fa = (a < (n1 + 1) / 2) ? a : a - n1;
    const int fb = (b < (n2 + 1) / 2) ? b : b - n2;
    const double k1 = 2.0 * 3.14159265358979323846 * (double)fa / ((double)n1 * d1);
    const double k2 = 2.0 * 3.14159265358979323846 * (double)fb / ((double)n2 * d2);
    const double kz = sqrt(fmax(k * k - k1 * k1 - k2 * k2, 0.0));
    const double th = (kz - k) * dz;
    double s, c, sh, ch;
    sincos(th, &s, &c);
    sincos(0.5 * th, &sh, &ch);
    hm1t[e] = make_float2((float)(-2.0 * sh * sh * inv), (float)(s * inv));
  }
}

// ------------------------------------------------------ in-place transforms
// The two passes at the other lengths (fft.cuh's in-place plans); the spectrum rows stay
// in the order of the plan's last stage, and the H table with them.  psi holds X_z =
// psi_z T_z in a step.
//
// Rows: a CTA owns rpc rows of one probe.  The inverse's last stage (the plan's first),
// the slice's own arithmetic and the forward transform's first stage share registers.
// 240 x 150, 32 probes: 58 -> 39 us per slice, adjoint 60 -> 39 (200 x 200, 50: 63 -> 57;
// 48 x 60, 64: 17 -> 12; 90 x 75, 16: 19 -> 15.5; what remains is issue and latency)
// against Stockham passes with radices up to 8 (a pass and a barrier per radix and
// direction, four more rounds through shared memory, no CTA for a remainder of rows).
template <int PHASE>
__global__ void __launch_bounds__(kMs3Threads, 2) ms3_mix_rows_kernel(const Ms3Params q, const __grid_constant__ MixPlan pl,
                                                                   int rpc, int z) {
  extern __shared__ __align__(16) float2 fsm[];
  const int n = pl.n, tid = threadIdx.x, row0 = blockIdx.x * rpc;
  const int tot = min(rpc, q.n1 - row0) * n;
  float2 *tw = fsm, *buf = tw + pl.tw_total;
  const size_t pbase = (size_t)blockIdx.y * q.N;
  const int g0 = row0 * n;  // first element of the CTA's rows within the slice
  constexpr bool STEP = PHASE == kMs3FwdStep || PHASE == kMs3BwdStep;
  const bool last = PHASE == kMs3FwdStep ? z + 1 == q.L : PHASE == kMs3BwdStep && z == 0;
  pdl_trigger();
  for (int e = tid; e < pl.tw_total; e += kMs3Threads) cp_async8(&tw[e], &q.tw2[e]);
  pdl_wait();
  if (STEP) {
    for (int e = tid; e < tot; e += kMs3Threads) cp_async8(&buf[mix_pad(e)], &q.W[pbase + g0 + e]);
  }
  cp_async_wait_all();
  __syncthreads();
  if (STEP) {
    mix_run<16, 4>(pl, pl.stages - 1, tot, buf, tw, nullptr, tid, kMs3Threads);
    __syncthreads();
    for (int s = pl.stages - 2; s > 0; --s) {
      mix_run<16, 1>(pl, s, tot, buf, tw, nullptr, tid, kMs3Threads);
      __syncthreads();
    }
  }
  const float2 *T = q.trans + (size_t)(PHASE == kMs3FwdStep ? (last ? z : z + 1) : z) * q.N + g0;
  const float2 *uf = PHASE == kMs3BwdStep ? q.u_fwd + ((size_t)blockIdx.y * q.nz + z) * q.N + g0 : nullptr;
  const float2 *in = (PHASE == kMs3FwdStart ? q.probes : q.src_exit) + pbase + g0;
  float2 *psi = q.psi + pbase + g0, *ex = q.exit_out ? q.exit_out + pbase + g0 : nullptr;
  float2 *us = q.u_store ? q.u_store + ((size_t)blockIdx.y * q.nz + (STEP ? z + 1 : 0)) * q.N + g0 : nullptr;
  mix_radix<16>(pl.radix[0], [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const int str = pl.str[0];
    for (int u = tid; u < tot / R; u += kMs3Threads) {
      const int b = fast_div(u, pl.ms[0]), t = u - b * str, base = b * n + t;
      const float2 *w = tw + t;
      float2 v[16], pz[R], tz[R], uz[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int e = base + r * str;
        if (STEP) pz[r] = psi[e];
        else v[r] = in[e];
        if (PHASE != kMs3BwdStart) tz[r] = T[e];
        if (PHASE == kMs3BwdStep) uz[r] = __ldcs(&uf[e]);
      }
      if (STEP) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          v[r] = buf[mix_pad(base + r * str)];
          if (r > 0) v[r] = cmulc(v[r], w[r * str]);
        }
        mix_dft<R>(v, 1.f);
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int e = base + r * str;
        if (PHASE == kMs3FwdStart || PHASE == kMs3FwdStep) {
          // psi_{z+1} = X_z + IFFT2((H-1) FFT2 X_z), X_{z+1} = psi_{z+1} T_{z+1}
          if (STEP) v[r] = cadd(pz[r], v[r]);
          if (us) __stcs(&us[e], v[r]);
          if (last) {
            if (ex) ex[e] = v[r];
          } else {
            v[r] = cfma(tz[r], v[r], v[r]);
          }
        } else if (PHASE == kMs3BwdStep) {
          // g_z = lambda_{z+1} + IFFT2(conj(H-1) FFT2 lambda_{z+1});
          // grad_t[z] += g_z conj(T_z u_z);  lambda_z = conj(T_z) g_z
          const float2 gv = cadd(pz[r], v[r]);
          red_add_cx(q.grad_t + (size_t)z * q.N + g0 + e, cmulc(gv, cfma(tz[r], uz[r], uz[r])));
          v[r] = cadd(gv, cmulc(gv, tz[r]));
        }
        if (!last) psi[e] = v[r];
      }
      if (last) continue;
      mix_dft<R>(v, -1.f);
#pragma unroll
      for (int r = 0; r < R; ++r) buf[mix_pad(base + r * str)] = r ? cmul(v[r], w[r * str]) : v[0];
    }
  });
  if (last) return;
  __syncthreads();
  for (int s = 1; s + 1 < pl.stages; ++s) {
    mix_run<16, 0>(pl, s, tot, buf, tw, nullptr, tid, kMs3Threads);
    __syncthreads();
  }
  mix_run<16, 3>(pl, pl.stages - 1, tot, buf, tw, nullptr, tid, kMs3Threads);
  __syncthreads();
  for (int e = tid; e < tot; e += kMs3Threads) q.W[pbase + g0 + e] = buf[mix_pad(e)];
}

// Columns: a CTA owns 2^lc columns of one probe (the last one fewer), place i of column c
// at i 2^lc + c in shared memory: every access runs along c.  The first stage reads and
// the last one writes W directly.
template <bool CONJ>
__global__ void __launch_bounds__(kMs3Threads) ms3_mix_cols_kernel(const Ms3Params q, const __grid_constant__ MixPlan pl,
                                                                   int lc) {
  extern __shared__ __align__(16) float2 fsm[];
  const int n = pl.n, w = q.n2, tid = threadIdx.x, C = 1 << lc, c = tid & (C - 1);  // kMs3Threads is a multiple of C
  const int col = (blockIdx.x << lc) + c;
  const bool ok = col < w;
  float2 *tw = fsm, *buf = tw + pl.tw_total + c;
  float2 *base = q.W + (size_t)blockIdx.y * q.N + col;
  const float2 *h = q.hm1t + col;
  pdl_trigger();
  for (int e = tid; e < pl.tw_total; e += kMs3Threads) cp_async8(&tw[e], &q.tw1[e]);
  cp_async_wait_all();
  __syncthreads();
  pdl_wait();
  // stage s; KIND 0: forward, 1: inverse, 2: last forward, product and inverse; GLOBAL:
  // the plan's first stage, W instead of shared memory on its outer side
  auto run = [&](auto kind, auto global, int s) {
    constexpr int KIND = decltype(kind)::value;
    constexpr bool GLOBAL = decltype(global)::value;
    mix_radix<16>(pl.radix[s], [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      const int str = pl.str[s];
      for (int u = tid >> lc; u < n / R; u += kMs3Threads >> lc) {
        const int b = fast_div(u, pl.ms[s]), t = u - b * str, at = b * (R * str) + t;
        const float2 *tws = tw + pl.tw[s] + t;
        float2 v[16], hv[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int i = at + r * str;
          if (GLOBAL && KIND == 0) v[r] = ok ? base[(size_t)i * w] : make_float2(0.f, 0.f);
          else v[r] = buf[i << lc];
          if (KIND == 1 && r > 0) v[r] = cmulc(v[r], tws[r * str]);
          if (KIND == 2) hv[r] = ok ? h[(size_t)i * w] : make_float2(0.f, 0.f);
        }
        mix_dft<R>(v, KIND == 1 ? 1.f : -1.f);
        if (KIND == 2) {
#pragma unroll
          for (int r = 0; r < R; ++r) v[r] = CONJ ? cmulc(v[r], hv[r]) : cmul(v[r], hv[r]);
          mix_dft<R>(v, 1.f);
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int i = at + r * str;
          if (KIND == 0 && r > 0) v[r] = cmul(v[r], tws[r * str]);
          if (GLOBAL && KIND == 1) {
            if (ok) base[(size_t)i * w] = v[r];
          } else {
            buf[i << lc] = v[r];
          }
        }
      }
    });
  };
  using std::integral_constant;
  using std::bool_constant;
  run(integral_constant<int, 0>{}, bool_constant<true>{}, 0);
  __syncthreads();
  for (int s = 1; s + 1 < pl.stages; ++s) {
    run(integral_constant<int, 0>{}, bool_constant<false>{}, s);
    __syncthreads();
  }
  run(integral_constant<int, 2>{}, bool_constant<false>{}, pl.stages - 1);
  __syncthreads();
  for (int s = pl.stages - 2; s > 0; --s) {
    run(integral_constant<int, 1>{}, bool_constant<false>{}, s);
    __syncthreads();
  }
  run(integral_constant<int, 1>{}, bool_constant<true>{}, 0);
}

// ------------------------------------------------ register four-step kernels
// The two passes for row and column lengths 64, 128, 192 and 256 (R1 R2) with
// the transforms in registers (fft.cuh): 256 threads, 256 / R1 rows or columns per
// CTA.  The row kernel's inverse transform ends with the field's elements in the
// registers where the next forward transform starts, so the multiplication by T and
// everything else between the two happens there, and an element crosses shared memory
// once per transform.  The psi buffer holds X_z = psi_z T_z here (psi_{z+1} = X_z +
// update needs no T_z).  Stockham passes in shared memory were bound by it
// (73-83 % of its throughput); a slice of 64 probes of 256 x 256 took 95 us with them
// (adjoint 99) and takes 43 us (48) with these.
template <int R1, int R2, int PHASE>
__global__ void __launch_bounds__(256, 2) ms3_rows4_kernel(const Ms3Params q, const float2 *__restrict__ twg, int z) {
  constexpr int N = R1 * R2, RPC = 256 / R1, S = R1 * (R2 + 1);
  __shared__ float2 buf[RPC * S];
  __shared__ float2 tw[R1 * (R2 + 1)];
  const int pr = blockIdx.y, tid = threadIdx.x;
  const size_t pbase = (size_t)pr * q.N;
  const int g0 = blockIdx.x * RPC * N;
  pdl_trigger();
  for (int e = tid; e < R1 * (R2 + 1); e += 256) tw[e] = twg[e];
  const int ra = tid / R2, n2 = tid % R2;  // stage A: (row, n2), element R2 n1 + n2
  const int rc = tid / R1, k1 = tid % R1;  // stage C: (row, k1), frequency k1 + R1 k2
  const bool inA = tid < RPC * R2;
  const int ga = g0 + ra * N + n2;
  float2 *wrow = q.W + pbase + g0 + rc * N + k1;
  const bool last = PHASE == kMs3FwdStep && z + 1 == q.L;
  float2 x[16], pz[R1], tz[R1], uz[R1];
  if (PHASE == kMs3FwdStart || PHASE == kMs3BwdStart) {
    __syncthreads();
    if (inA) {
#pragma unroll
      for (int j = 0; j < R1; ++j) {
        const int g = ga + R2 * j;
        float2 v = (PHASE == kMs3FwdStart ? q.probes : q.src_exit)[pbase + g];
        if (PHASE == kMs3FwdStart) {
          if (q.u_store) q.u_store[(size_t)pr * q.nz * q.N + g] = v;
          v = cfma(q.trans[g], v, v);
        }
        q.psi[pbase + g] = v;
        x[j] = v;
      }
    }
  } else {
    // The adjoint's third and fourth operands at 192 and 256 wait until the field is in x:
    // held from the start they spilled (64 probes, 256 x 256: 51.5 -> 47.4 us per slice, 192 x
    // 192: 33.6 -> 31.2;
    // 128 x 128 is faster with them early, 16.1 against 16.4).
    constexpr bool LATE = PHASE == kMs3BwdStep && R2 > 8;
    const float2 *T = q.trans + (size_t)(PHASE == kMs3FwdStep ? (last ? z : z + 1) : z) * q.N;
    const float2 *u = PHASE == kMs3BwdStep ? q.u_fwd + ((size_t)pr * q.nz + z) * q.N : nullptr;
    if (inA && !LATE) {  // what no kernel of the march writes, before the column pass is complete
#pragma unroll
      for (int j = 0; j < R1; ++j) {
        tz[j] = T[ga + R2 * j];
        if (PHASE == kMs3BwdStep) uz[j] = __ldcs(&u[ga + R2 * j]);
      }
    }
    pdl_wait();
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) x[k2] = wrow[R1 * k2];
    auto load_psi = [&]() {
#pragma unroll
      for (int j = 0; j < R1; ++j) pz[j] = q.psi[pbase + ga + R2 * j];
    };
    if (inA && !LATE) load_psi();
    dft_reg<R2>(x, 1.f);
    __syncthreads();  // the twiddles are in place
#pragma unroll
    for (int m = 0; m < R2; ++m)
      buf[rc * S + k1 * (R2 + 1) + m] = m ? cmulc(x[m], tw[k1 * (R2 + 1) + m]) : x[0];
    if (inA && LATE) load_psi();
    __syncthreads();
    if (inA) {
#pragma unroll
      for (int k = 0; k < R1; ++k) x[k] = buf[ra * S + k * (R2 + 1) + n2];
      dft_reg<R1>(x, 1.f);
#pragma unroll
      for (int j = 0; j < R1; ++j) x[j] = cadd(pz[j], x[j]);
      if (LATE) {
#pragma unroll
        for (int j = 0; j < R1; ++j) {
          tz[j] = T[ga + R2 * j];
          uz[j] = __ldcs(&u[ga + R2 * j]);
        }
      }
      if (PHASE == kMs3FwdStep) {
        // psi_{z+1} = X_z + IFFT2((H-1) FFT2 X_z), X_{z+1} = psi_{z+1} T_{z+1}
        float2 *us = q.u_store ? q.u_store + ((size_t)pr * q.nz + z + 1) * q.N + ga : nullptr;
#pragma unroll
        for (int j = 0; j < R1; ++j) {
          const float2 v = x[j];
          if (us) __stcs(&us[R2 * j], v);
          if (last) {
            if (q.exit_out) q.exit_out[pbase + ga + R2 * j] = v;
          } else {
            x[j] = cfma(tz[j], v, v);
            q.psi[pbase + ga + R2 * j] = x[j];
          }
        }
      } else {
        // g_z = lambda_{z+1} + IFFT2(conj(H-1) FFT2 lambda_{z+1});
        // grad_t[z] += g_z conj(T_z u_z);  lambda_z = conj(T_z) g_z
        float2 *gt = q.grad_t + (size_t)z * q.N + ga;
#pragma unroll
        for (int j = 0; j < R1; ++j) {
          const float2 gv = x[j];
          red_add_cx(gt + R2 * j, cmulc(gv, cfma(tz[j], uz[j], uz[j])));
          x[j] = cadd(gv, cmulc(gv, tz[j]));
          if (z > 0) q.psi[pbase + ga + R2 * j] = x[j];
        }
      }
    }
    if (last || (PHASE == kMs3BwdStep && z == 0)) return;
  }
  if (inA) {  // (in a step, into the slots that this thread has just read)
    dft_reg<R1>(x, -1.f);
#pragma unroll
    for (int k = 0; k < R1; ++k)
      buf[ra * S + k * (R2 + 1) + n2] = k ? cmul(x[k], tw[k * (R2 + 1) + n2]) : x[0];
  }
  __syncthreads();
#pragma unroll
  for (int m = 0; m < R2; ++m) x[m] = buf[rc * S + k1 * (R2 + 1) + m];
  dft_reg<R2>(x, -1.f);
#pragma unroll
  for (int k2 = 0; k2 < R2; ++k2) wrow[R1 * k2] = x[k2];
}

// Column pass (hm1t by rows).  Grid (n2 / CPC, P).
template <int R1, int R2, bool CONJ>
__global__ void __launch_bounds__(256, 3) ms3_cols4_kernel(const Ms3Params q, const float2 *__restrict__ twg) {
  constexpr int N = R1 * R2, CPC = 256 / R1;
  __shared__ float2 buf[N * CPC];  // [k1][n2][c]
  __shared__ float2 tw[R1 * (R2 + 1)];
  const int tid = threadIdx.x, w = q.n2;
  pdl_trigger();
  for (int e = tid; e < R1 * (R2 + 1); e += 256) tw[e] = twg[e];
  const int c = tid % CPC, n2 = tid / CPC;  // stage A: (c, n2); stage C: (c, k1)
  const int k1 = n2;
  const bool inA = n2 < R2;
  float2 *base = q.W + (size_t)blockIdx.y * q.N + blockIdx.x * CPC + c;
  const float2 *h = q.hm1t + blockIdx.x * CPC + c + (size_t)k1 * w;
  float2 x[16], hv[R2];
#pragma unroll
  for (int k2 = 0; k2 < R2; ++k2) hv[k2] = h[(size_t)R1 * k2 * w];
  pdl_wait();
  if (inA) {
#pragma unroll
    for (int j = 0; j < R1; ++j) x[j] = base[(size_t)(R2 * j + n2) * w];
    dft_reg<R1>(x, -1.f);
  }
  __syncthreads();
  if (inA) {
#pragma unroll
    for (int k = 0; k < R1; ++k) buf[(k * R2 + n2) * CPC + c] = k ? cmul(x[k], tw[k * (R2 + 1) + n2]) : x[0];
  }
  __syncthreads();
#pragma unroll
  for (int m = 0; m < R2; ++m) x[m] = buf[(k1 * R2 + m) * CPC + c];
  dft_reg<R2>(x, -1.f);
#pragma unroll
  for (int k2 = 0; k2 < R2; ++k2) x[k2] = CONJ ? cmulc(x[k2], hv[k2]) : cmul(x[k2], hv[k2]);
  dft_reg<R2>(x, 1.f);
  // this thread's own slots: no other thread reads (k1, ., c) before the barrier
#pragma unroll
  for (int m = 0; m < R2; ++m) buf[(k1 * R2 + m) * CPC + c] = m ? cmulc(x[m], tw[k1 * (R2 + 1) + m]) : x[0];
  __syncthreads();
  if (inA) {
#pragma unroll
    for (int k = 0; k < R1; ++k) x[k] = buf[(k * R2 + n2) * CPC + c];
    dft_reg<R1>(x, 1.f);
#pragma unroll
    for (int j = 0; j < R1; ++j) base[(size_t)(R2 * j + n2) * w] = x[j];
  }
}

// The padded twiddle table W_N^{n2 k1} at k1 (R2 + 1) + n2.
__global__ void ms3_twiddle4_kernel(int r1, int r2, float2 *tw) {
  for (int e = threadIdx.x; e < r1 * (r2 + 1); e += blockDim.x) {
    const int k1 = e / (r2 + 1), n2 = e % (r2 + 1);
    double sv, cv;
    sincospi(-2.0 * (double)(k1 * n2) / (double)(r1 * r2), &sv, &cv);
    tw[e] = make_float2((float)cv, (float)sv);
  }
}

using Ms3Rows4 = void (*)(const Ms3Params, const float2 *, int);
using Ms3Cols4 = void (*)(const Ms3Params, const float2 *);
template <int PHASE>
static Ms3Rows4 pick_rows4(int n) {
  switch (n) {
    case 64: return ms3_rows4_kernel<8, 8, PHASE>;
    case 128: return ms3_rows4_kernel<16, 8, PHASE>;
    case 192: return ms3_rows4_kernel<16, 12, PHASE>;
    default: return ms3_rows4_kernel<16, 16, PHASE>;
  }
}
template <bool CONJ>
static Ms3Cols4 pick_cols4(int n) {
  switch (n) {
    case 64: return ms3_cols4_kernel<8, 8, CONJ>;
    case 128: return ms3_cols4_kernel<16, 8, CONJ>;
    case 192: return ms3_cols4_kernel<16, 12, CONJ>;
    default: return ms3_cols4_kernel<16, 16, CONJ>;
  }
}

struct Ms3Work {
  float2 *psi, *W, *hm1t, *tw1, *tw2;
  size_t bytes;
};

static size_t a256(size_t b) { return (b + 255) & ~(size_t)255; }

static Ms3Work ms3_layout(char *base, int n1, int n2, int P) {
  Ms3Work w{};
  size_t off = 0;
  auto take = [&](size_t bytes) {
    float2 *p = base ? reinterpret_cast<float2 *>(base + off) : nullptr;
    off += a256(bytes);
    return p;
  };
  const size_t N = (size_t)n1 * n2;
  w.psi = take((size_t)P * N * sizeof(float2));
  w.W = take((size_t)P * N * sizeof(float2));
  w.hm1t = take(N * sizeof(float2));
  // room for either kernels' tables (in-place plans: at most 1.3 n)
  w.tw1 = take((size_t)(n1 + n1 / 2 + 16) * sizeof(float2));
  w.tw2 = take((size_t)(n2 + n2 / 2 + 16) * sizeof(float2));
  w.bytes = off;
  return w;
}

static int ms3_check_op(const tp_ms3d_op *op) {
  if (op == nullptr) return set_error(TP_ERR_INVALID, "op is NULL");
  if (op->nz < 2) return set_error(TP_ERR_INVALID, "nz=%d must be >= 2", op->nz);
  if (make_fft_plan(op->n1).npass == 0 || make_fft_plan(op->n2).npass == 0)
    return set_error(TP_ERR_UNSUPPORTED, "3D multislice grid %d x %d: each side must be 2^a 3^b 5^c <= %d", op->n1,
                     op->n2, kFftMaxN);
  if (!(op->k > 0.0) || !(op->d1 > 0.0) || !(op->d2 > 0.0))
    return set_error(TP_ERR_INVALID, "k, d1, d2 must be positive");
  return TP_OK;
}

// Runs the forward march (backward = false) or the adjoint march.
static int ms3_run(const tp_ms3d_op *op, Ms3Params q, bool backward, void *workspace, size_t workspace_bytes,
                   cudaStream_t st) {
  const int n1 = op->n1, n2 = op->n2;
  if (workspace == nullptr || (reinterpret_cast<uintptr_t>(workspace) & 255u) != 0)
    return set_error(TP_ERR_INVALID, "3D multislice workspace must be non-NULL and 256-byte aligned");
  Ms3Work w = ms3_layout(static_cast<char *>(workspace), n1, n2, q.P);
  if (workspace_bytes < w.bytes)
    return set_error(TP_ERR_WORKSPACE, "3D multislice workspace %zu B < %zu B", workspace_bytes, w.bytes);
  q.psi = w.psi;
  q.W = w.W;
  q.hm1t = w.hm1t;
  q.tw1 = w.tw1;
  q.tw2 = w.tw2;
  // register four-step kernels where the length has a plan and the other axis
  // splits into whole CTAs
  const bool four_r = four_step_size(n2) && n1 % (256 / four_r1(n2)) == 0;
  const bool four_c = four_step_size(n1) && n2 % (256 / four_r1(n1)) == 0;
  const MixPlan p1 = four_c ? MixPlan{} : make_mix_plan(n1), p2 = four_r ? MixPlan{} : make_mix_plan(n2);
  if (four_c) ms3_twiddle4_kernel<<<1, 256, 0, st>>>(four_r1(n1), four_r2(n1), w.tw1);
  else ms3_twiddle_mix_kernel<<<(n1 + 255) / 256, 256, 0, st>>>(p1, w.tw1);
  if (four_r) ms3_twiddle4_kernel<<<1, 256, 0, st>>>(four_r1(n2), four_r2(n2), w.tw2);
  else ms3_twiddle_mix_kernel<<<(n2 + 255) / 256, 256, 0, st>>>(p2, w.tw2);
  ms3_kernel_h_kernel<<<(q.N + 255) / 256 < 1184 ? (q.N + 255) / 256 : 1184, 256, 0, st>>>(
      n1, n2, p1, p2, w.tw1, w.tw2, (four_c ? four_dft_gain(n1) : mix_dft_gain(p1)) + (four_r ? four_dft_gain(n2) : mix_dft_gain(p2)),
      op->k, op->d1, op->d2, op->dz, w.hm1t);
  TP_CHECK_CUDA(cudaGetLastError());
  // in-place kernels: rows and columns per CTA, about 4096 elements
  int rpc = 4096 / n2 < 16 ? 4096 / n2 : 16, lc = 4;
  if (rpc < 1) rpc = 1;
  while (lc > 0 && (n1 << lc) > 4096) --lc;
  const size_t smem_r = (size_t)(p2.tw_total + mix_pad(rpc * n2) + 1) * sizeof(float2);
  const size_t smem_c = (size_t)(p1.tw_total + (n1 << lc)) * sizeof(float2);
  const auto start_m = backward ? ms3_mix_rows_kernel<kMs3BwdStart> : ms3_mix_rows_kernel<kMs3FwdStart>;
  const auto step_m = backward ? ms3_mix_rows_kernel<kMs3BwdStep> : ms3_mix_rows_kernel<kMs3FwdStep>;
  const auto cols_m = backward ? ms3_mix_cols_kernel<true> : ms3_mix_cols_kernel<false>;
  if (!four_r) {
    TP_CHECK_CUDA(cudaFuncSetAttribute(start_m, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_r));
    TP_CHECK_CUDA(cudaFuncSetAttribute(step_m, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_r));
  }
  if (!four_c) TP_CHECK_CUDA(cudaFuncSetAttribute(cols_m, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_c));
  const dim3 gr((n1 + rpc - 1) / rpc, q.P), gc((n2 + (1 << lc) - 1) >> lc, q.P);
  const dim3 gr4(four_r ? n1 / (256 / four_r1(n2)) : 1, q.P), gc4(four_c ? n2 / (256 / four_r1(n1)) : 1, q.P);
  const Ms3Rows4 start4 = backward ? pick_rows4<kMs3BwdStart>(n2) : pick_rows4<kMs3FwdStart>(n2);
  const Ms3Rows4 step4 = backward ? pick_rows4<kMs3BwdStep>(n2) : pick_rows4<kMs3FwdStep>(n2);
  const Ms3Cols4 cols4 = backward ? pick_cols4<true>(n1) : pick_cols4<false>(n1);
  // every pass but the first starts early (pdl_wait)
  auto row_pass = [&](bool start, int z) -> cudaError_t {
    if (four_r) return launch_dependent(start ? start4 : step4, gr4, dim3(256), 0, st, !start, q, w.tw2, z);
    return launch_dependent(start ? start_m : step_m, gr, dim3(kMs3Threads), smem_r, st, !start, q, p2, rpc, z);
  };
  TP_CHECK_CUDA(row_pass(true, backward ? q.L : 0));
  for (int t = 0; t < q.L; ++t) {
    if (four_c) TP_CHECK_CUDA(launch_dependent(cols4, gc4, dim3(256), 0, st, true, q, w.tw1));
    else TP_CHECK_CUDA(launch_dependent(cols_m, gc, dim3(kMs3Threads), smem_c, st, true, q, p1, lc));
    TP_CHECK_CUDA(row_pass(false, backward ? q.L - 1 - t : t));
  }
  return check_cuda(cudaGetLastError(), "ms3d march launch");
}

static Ms3Params ms3_params(const tp_ms3d_op *op, int P) {
  Ms3Params q{};
  q.n1 = op->n1;
  q.n2 = op->n2;
  q.N = op->n1 * op->n2;
  q.nz = op->nz;
  q.L = op->nz - 1;
  q.P = P;
  return q;
}

}  // namespace tp

using namespace tp;

extern "C" size_t tp_ms3d_workspace_bytes(int32_t n1, int32_t n2, int32_t num_probes) {
  if (n1 < 1 || n2 < 1 || num_probes < 1) return 0;
  return ms3_layout(nullptr, n1, n2, num_probes).bytes;
}

extern "C" int tp_ms3d_transmission(const tp_ms3d_op *op, const void *n_field, int32_t n_dtype, void *trans,
                                    tp_stream_t stream) {
  int rc = ms3_check_op(op);
  if (rc) return rc;
  if (!n_field || !trans) return set_error(TP_ERR_INVALID, "n_field/trans is NULL");
  return ms_transmission_launch(op->n1 * op->n2, op->nz, op->k, op->dz, op->n_medium[0], op->n_medium[1], n_field,
                                n_dtype, static_cast<float2 *>(trans), reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int tp_ms3d_march(const tp_ms3d_op *op, const void *trans, const void *probes, int32_t num_probes,
                             void *u_store, void *exit_out, void *workspace, size_t workspace_bytes,
                             tp_stream_t stream) {
  int rc = ms3_check_op(op);
  if (rc) return rc;
  if (!trans || !probes || num_probes < 1) return set_error(TP_ERR_INVALID, "bad 3D multislice march args");
  Ms3Params q = ms3_params(op, num_probes);
  q.trans = static_cast<const float2 *>(trans);
  q.probes = static_cast<const float2 *>(probes);
  q.u_store = static_cast<float2 *>(u_store);
  q.exit_out = static_cast<float2 *>(exit_out);
  return ms3_run(op, q, false, workspace, workspace_bytes, reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int tp_ms3d_backward(const tp_ms3d_op *op, const void *trans, const void *u_fwd, const void *src_exit,
                                int32_t num_probes, void *grad_t, void *workspace, size_t workspace_bytes,
                                tp_stream_t stream) {
  int rc = ms3_check_op(op);
  if (rc) return rc;
  if (!trans || !u_fwd || !src_exit || !grad_t || num_probes < 1)
    return set_error(TP_ERR_INVALID, "bad 3D multislice backward args");
  Ms3Params q = ms3_params(op, num_probes);
  q.trans = static_cast<const float2 *>(trans);
  q.u_fwd = static_cast<const float2 *>(u_fwd);
  q.src_exit = static_cast<const float2 *>(src_exit);
  q.grad_t = static_cast<float2 *>(grad_t);
  return ms3_run(op, q, true, workspace, workspace_bytes, reinterpret_cast<cudaStream_t>(stream));
}
