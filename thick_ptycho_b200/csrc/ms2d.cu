// Batched 1D FFTs and far-field / amplitude-loss heads on the shared-memory FFT of
// fft.cuh, and the 2D multislice (angular-spectrum) march with its adjoint on register
// and in-place transforms.
//
// Replaces: numpy.fft in the far field (forward_model/base/base_solver.py:
// 234-242) and the phase-retrieval projection (reconstruction/
// base_reconstructor.py:171-207); the multislice solver's per-probe loop
// (forward_model/multislice/ms_solver.py:49-159).
#include <cuda_runtime.h>

#include <type_traits>

#include "fft.cuh"
#include "tp_errors.h"
#include "tpcuda.h"

namespace tp {

constexpr int kFftThreads = 256;

static int fft_rows_per_cta(int n) {
  int r = kFftMaxN / n;
  if (r > 8) r = 8;
  return r < 1 ? 1 : r;
}

// ------------------------------------------------------------------ 1D FFT
__global__ void __launch_bounds__(kFftThreads) fft1d_kernel(const FftPlan pl, int batch, const float2 *__restrict__ in,
                                                            float2 *__restrict__ out, int inverse, int rows) {
  extern __shared__ __align__(16) float2 fsm[];
  const int n = pl.n;
  float2 *tw = fsm, *a = fsm + n, *b = a + rows * n;
  const int r0 = blockIdx.x * rows;
  const int nb = min(rows, batch - r0);
  fft_twiddles(tw, n, threadIdx.x, blockDim.x);
  for (int e = threadIdx.x; e < nb * n; e += blockDim.x) a[e] = in[(size_t)r0 * n + e];
  __syncthreads();
  float2 *res = fft_block(a, b, pl, tw, inverse != 0, nb, threadIdx.x, blockDim.x);
  const float s = inverse ? 1.f / (float)n : 1.f;
  for (int e = threadIdx.x; e < nb * n; e += blockDim.x) {
    const float2 v = res[e];
    out[(size_t)r0 * n + e] = make_float2(v.x * s, v.y * s);
  }
}

// |FFT(exit)|^2 (intensity, unnormalised, no shift)
__global__ void __launch_bounds__(kFftThreads) farfield_kernel(const FftPlan pl, int batch, const float2 *__restrict__ in,
                                                               float *__restrict__ out, int rows) {
  extern __shared__ __align__(16) float2 fsm[];
  const int n = pl.n;
  float2 *tw = fsm, *a = fsm + n, *b = a + rows * n;
  const int r0 = blockIdx.x * rows;
  const int nb = min(rows, batch - r0);
  fft_twiddles(tw, n, threadIdx.x, blockDim.x);
  for (int e = threadIdx.x; e < nb * n; e += blockDim.x) a[e] = in[(size_t)r0 * n + e];
  __syncthreads();
  float2 *res = fft_block(a, b, pl, tw, false, nb, threadIdx.x, blockDim.x);
  for (int e = threadIdx.x; e < nb * n; e += blockDim.x) {
    const float2 v = res[e];
    out[(size_t)r0 * n + e] = fmaf(v.x, v.x, v.y * v.y);
  }
}

// loss = sum (|F e| - a)^2 ;  grad = sum_k F^H[2 (|U|-a) U/|U|]  (torch convention)
__global__ void __launch_bounds__(kFftThreads) amp_residual_kernel(const FftPlan pl, int batch,
                                                                   const float2 *__restrict__ ex,
                                                                   const float *__restrict__ amp,
                                                                   float2 *__restrict__ grad, double *loss, int rows) {
  extern __shared__ __align__(16) float2 fsm[];
  __shared__ double red[kFftThreads / 32];
  const int n = pl.n;
  float2 *tw = fsm, *a = fsm + n, *b = a + rows * n;
  const int r0 = blockIdx.x * rows;
  const int nb = min(rows, batch - r0);
  fft_twiddles(tw, n, threadIdx.x, blockDim.x);
  for (int e = threadIdx.x; e < nb * n; e += blockDim.x) a[e] = ex[(size_t)r0 * n + e];
  __syncthreads();
  float2 *U = fft_block(a, b, pl, tw, false, nb, threadIdx.x, blockDim.x);
  double acc = 0.0;
  for (int e = threadIdx.x; e < nb * n; e += blockDim.x) {
    const float2 u = U[e];
    const double mag = sqrt((double)u.x * u.x + (double)u.y * u.y);
    const double d = mag - (double)amp[(size_t)r0 * n + e];
    acc += d * d;
    const float f = mag > 0.0 ? (float)(2.0 * d / mag) : 0.f;
    U[e] = make_float2(f * u.x, f * u.y);
  }
  __syncthreads();
  float2 *other = (U == a) ? b : a;
  float2 *G = fft_block(U, other, pl, tw, true, nb, threadIdx.x, blockDim.x);  // unnormalised inverse = F^H
  for (int e = threadIdx.x; e < nb * n; e += blockDim.x) grad[(size_t)r0 * n + e] = G[e];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < (int)(blockDim.x / 32); ++w) s += red[w];
    atomicAdd(loss, s);
  }
}

// ---------------------------------------------------------------- multislice
struct MsParams {
  int n, nz, L, P;
  double k, dx, dz;
  double nmr, nmi;  // medium index
  const void *field;
  int dtype;
  const float2 *trans;  // (L, n)
  const float2 *probes;
  float2 *u_store;  // (P, nz, n) or null
  float2 *exit_out;
  const float2 *u_fwd;   // backward: forward field (P, nz, n)
  const float2 *src_exit;
  float2 *grad_t;  // backward: (L, n) accumulator of sum_p conj(T_z u_z) g_z
};

// T_z[x] - 1 with T_z[x] = exp(i k (n[x,z] - n_medium) dz), z = 0..L-1
// (ms_solver.py:86-88).  The table holds the deviation from one, computed in
// fp64 (expm1, -2 sin^2): T is 1 + O(k dn dz) and rounding it to fp32 every
// slice would bias the march.
__global__ void ms_transmission_kernel(const MsParams q, float2 *__restrict__ trans) {
  const size_t total = (size_t)q.L * q.n;
  for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
    const int x = (int)(idx % q.n), z = (int)(idx / q.n);
    double nr, ni;
    if (q.dtype == TP_C128) {
      const double2 v = static_cast<const double2 *>(q.field)[(size_t)x * q.nz + z];
      nr = v.x;
      ni = v.y;
    } else {
      const float2 v = static_cast<const float2 *>(q.field)[(size_t)x * q.nz + z];
      nr = v.x;
      ni = v.y;
    }
    const double ph = q.k * (nr - q.nmr) * q.dz, am1 = expm1(-q.k * (ni - q.nmi) * q.dz);
    double s, c, sh, ch;
    sincos(ph, &s, &c);
    sincos(0.5 * ph, &sh, &ch);
    // e^a (c + i s) - 1 = (e^a - 1) c + (c - 1) + i e^a s,  c - 1 = -2 sin^2(ph/2)
    trans[idx] = make_float2((float)(am1 * c - 2.0 * sh * sh), (float)((am1 + 1.0) * s));
  }
}

// (H[j] - 1) scale with H[j] = exp(i (kz - k) dz), kz = sqrt(max(k^2 - kx^2, 0)),
// kx = 2 pi fftfreq(n, dx) (ms_solver.py:49-72); fp64, kept as the deviation
// from one like the transmission.
__device__ __forceinline__ float2 ms_h_minus_1(const MsParams &q, int j, double scale) {
  const int f = (j < (q.n + 1) / 2) ? j : j - q.n;
  const double kx = 2.0 * 3.14159265358979323846 * (double)f / ((double)q.n * q.dx);
  const double kz = sqrt(fmax(q.k * q.k - kx * kx, 0.0));
  const double th = (kz - q.k) * q.dz;
  double s, c, sh, ch;
  sincos(th, &s, &c);
  sincos(0.5 * th, &sh, &ch);
  return make_float2((float)(-2.0 * sh * sh * scale), (float)(s * scale));
}
// Each slice is evaluated in delta form,
//   X = psi + (T_z - 1) psi,   psi' = X + IFFT((H - 1) . FFT(X)),
// so the FFT round-off scales with the small update instead of the field (the same
// reason the CN march keeps "1 + eps" coefficients); the adjoint: g = lambda +
// IFFT(conj(H - 1) . FFT(lambda)), grad_t[z] += sum_p g conj(T_z u_z), lambda <-
// conj(T_z) g, from lambda = src_exit at the exit plane.

// ------------------------------------------- register transforms, n = 16 R2 R3
// The march at n = 512, 1024, 2048 and 4096 with one probe per CTA of n / 16
// threads: a thread keeps 16 field values, and each transform is a radix-16, a
// radix-R2 and a radix-R3 step in registers with two shared-memory exchanges.  The
// forward transform leaves the spectrum in the order of its last step, where it is
// multiplied by H - 1 (kept in that order) and the inverse starts, so no pass only
// reorders; a thread's twiddles and its part of H are the same for every slice and
// stay in registers.  With index x = t + (n/16) j, t = a + R3 b and frequency
// k = k1 + 16 k2 + 16 R2 k3:
//   step 1 (thread t):       DFT-16 over j -> k1, times W_n^{t k1}
//   step 2 (unit (k1, a)):   DFT-R2 over b -> k2, times W_{n/16}^{a k2}
//   step 3 (unit (k1, k2)):  DFT-R3 over a -> k3
// and the inverse in the opposite order with conjugate twiddles.  The exchanges are
// padded so that neither side has bank conflicts, and alternate between two buffers
// (one barrier each).  T - 1 (and the adjoint's u) of the next slice arrive by
// asynchronous copies into the thread's own slots.  What remains is the latency of
// a slice's dependent steps: n = 2048, 64 probes, 1023 slices: forward with the field
// kept 13.7 -> 1.65 ms, adjoint 13.5 -> 2.30 ms against Stockham passes in shared memory.
template <int R2, int R3>
struct RegFft {
  static constexpr int N = 16 * R2 * R3, T = N / 16, M2 = 16 / R2, M3 = 16 / R3;
  static constexpr int S1 = T + R3, S2 = ((R2 * (R3 + 1) + 15) / 16) * 16 + R3;
  static constexpr int BUF = 16 * (S1 > S2 ? S1 : S2);
  float2 tw1[15], tw2[M2][R2 - 1], h[16];

  __device__ __forceinline__ static float2 root(int num, int den) {  // exp(-2 pi i num / den)
    double s, c;
    sincospi(-2.0 * (double)num / (double)den, &s, &c);
    return make_float2((float)c, (float)s);
  }
  __device__ __forceinline__ void init(const MsParams &q) {
    const int v = threadIdx.x;
#pragma unroll
    for (int k = 1; k < 16; ++k) tw1[k - 1] = root(v * k, N);
#pragma unroll
    for (int m = 0; m < M2; ++m) {
      const int a = (v + T * m) % R3;
#pragma unroll
      for (int k = 1; k < R2; ++k) tw2[m][k - 1] = root(a * k, T);
    }
    __shared__ double red[32];
    double g = 0.0;
#pragma unroll
    for (int k = 0; k < 15; ++k) g += modulus_less_1(tw1[k]);
#pragma unroll
    for (int m = 0; m < M2; ++m)
#pragma unroll
      for (int k = 0; k < R2 - 1; ++k) g += modulus_less_1(tw2[m][k]);
    g = cta_sum(g, red) / N + (dft_gain(16) + dft_gain(R2) + dft_gain(R3));
    const double scale = 1.0 / (N * (1.0 + g));
    // (H - 1) / n of this thread's frequencies, less the transforms' gain
#pragma unroll
    for (int m = 0; m < M3; ++m) {
      const int p = v + T * m, k1 = p / R2, k2 = p % R2;
#pragma unroll
      for (int k3 = 0; k3 < R3; ++k3) {
        h[m * R3 + k3] = ms_h_minus_1(q, k1 + 16 * k2 + 16 * R2 * k3, scale);
      }
    }
  }
  template <int R>
  __device__ __forceinline__ static void dft(float2 *x, float sign) {
    float2 w[16];
#pragma unroll
    for (int i = 0; i < R; ++i) w[i] = x[i];
    dft_reg<R>(w, sign);
#pragma unroll
    for (int i = 0; i < R; ++i) x[i] = w[i];
  }
  // x (x[j] at index threadIdx.x + T j) <- IFFT(h . FFT(x)), h conjugated for CONJ
  template <bool CONJ>
  __device__ __forceinline__ void apply(float2 (&x)[16], float2 *b0, float2 *b1) const {
    const int v = threadIdx.x;
    dft<16>(x, -1.f);
#pragma unroll
    for (int k = 0; k < 16; ++k) b0[k * S1 + v] = k ? cmul(x[k], tw1[k - 1]) : x[0];
    __syncthreads();
#pragma unroll
    for (int m = 0; m < M2; ++m) {
      const int u = v + T * m, k1 = u / R3, a = u % R3;
#pragma unroll
      for (int b = 0; b < R2; ++b) x[m * R2 + b] = b0[k1 * S1 + a + R3 * b];
      dft<R2>(x + m * R2, -1.f);
#pragma unroll
      for (int k = 0; k < R2; ++k)
        b1[k1 * S2 + k * (R3 + 1) + a] = k ? cmul(x[m * R2 + k], tw2[m][k - 1]) : x[m * R2];
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < M3; ++m) {
      const int p = v + T * m, k1 = p / R2, k2 = p % R2;
      float2 *c = b1 + k1 * S2 + k2 * (R3 + 1);  // this unit's own slots in both directions
#pragma unroll
      for (int a = 0; a < R3; ++a) x[m * R3 + a] = c[a];
      dft<R3>(x + m * R3, -1.f);
#pragma unroll
      for (int k = 0; k < R3; ++k)
        x[m * R3 + k] = CONJ ? cmulc(x[m * R3 + k], h[m * R3 + k]) : cmul(x[m * R3 + k], h[m * R3 + k]);
      dft<R3>(x + m * R3, 1.f);
#pragma unroll
      for (int a = 0; a < R3; ++a) c[a] = x[m * R3 + a];
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < M2; ++m) {
      const int u = v + T * m, k1 = u / R3, a = u % R3;
#pragma unroll
      for (int k = 0; k < R2; ++k) {
        const float2 w = b1[k1 * S2 + k * (R3 + 1) + a];
        x[m * R2 + k] = k ? cmulc(w, tw2[m][k - 1]) : w;
      }
      dft<R2>(x + m * R2, 1.f);
#pragma unroll
      for (int b = 0; b < R2; ++b) b0[k1 * S1 + a + R3 * b] = x[m * R2 + b];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const float2 w = b0[k * S1 + v];
      x[k] = k ? cmulc(w, tw1[k - 1]) : w;
    }
    dft<16>(x, 1.f);
  }
};

template <int R2, int R3>
static constexpr size_t ms_reg_smem(int streams) {
  return (size_t)(2 * RegFft<R2, R3>::BUF + 2 * streams * RegFft<R2, R3>::N) * sizeof(float2);
}

template <int R2, int R3>
__global__ void __launch_bounds__(RegFft<R2, R3>::T) ms_reg_march_kernel(const MsParams q) {
  using F = RegFft<R2, R3>;
  constexpr int N = F::N, T = F::T;
  extern __shared__ __align__(16) float2 fsm[];
  float2 *b0 = fsm, *b1 = b0 + F::BUF, *ts = b1 + F::BUF;  // ts: [2][N]
  const int v = threadIdx.x;
  const size_t p = blockIdx.x;
  auto stage = [&](int z) {
#pragma unroll
    for (int j = 0; j < 16; ++j) cp_async8(&ts[(z & 1) * N + v + T * j], &q.trans[(size_t)z * N + v + T * j]);
  };
  stage(0);
  cp_async_commit();
  F f;
  f.init(q);
  float2 X[16], y[16];
  float2 *store = q.u_store ? q.u_store + p * q.nz * N + v : nullptr;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    X[j] = q.probes[p * N + v + T * j];
    if (store) store[T * j] = X[j];
  }
  for (int z = 0; z < q.L; ++z) {
    if (z + 1 < q.L) stage(z + 1);
    cp_async_commit();
    cp_async_wait<1>();  // this thread's part of slice z
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      X[j] = cfma(ts[(z & 1) * N + v + T * j], X[j], X[j]);
      y[j] = X[j];
    }
    f.template apply<false>(y, b0, b1);
    if (store) store += N;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      X[j] = cadd(X[j], y[j]);
      if (store) __stcs(&store[T * j], X[j]);
    }
  }
  if (q.exit_out) {
#pragma unroll
    for (int j = 0; j < 16; ++j) q.exit_out[p * N + v + T * j] = X[j];
  }
}

template <int R2, int R3>
__global__ void __launch_bounds__(RegFft<R2, R3>::T) ms_reg_backward_kernel(const MsParams q) {
  using F = RegFft<R2, R3>;
  constexpr int N = F::N, T = F::T;
  extern __shared__ __align__(16) float2 fsm[];
  float2 *b0 = fsm, *b1 = b0 + F::BUF, *ts = b1 + F::BUF, *us = ts + 2 * N;  // ts, us: [2][N]
  const int v = threadIdx.x;
  const size_t p = blockIdx.x;
  auto stage = [&](int z) {
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      cp_async8(&ts[(z & 1) * N + v + T * j], &q.trans[(size_t)z * N + v + T * j]);
      cp_async8(&us[(z & 1) * N + v + T * j], &q.u_fwd[(p * q.nz + z) * N + v + T * j]);
    }
  };
  stage(q.L - 1);
  cp_async_commit();
  F f;
  f.init(q);
  float2 X[16], y[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) X[j] = q.src_exit[p * N + v + T * j];
  for (int z = q.L - 1; z >= 0; --z) {
    if (z > 0) stage(z - 1);
    cp_async_commit();
#pragma unroll
    for (int j = 0; j < 16; ++j) y[j] = X[j];
    f.template apply<true>(y, b0, b1);
    cp_async_wait<1>();
    float2 *grad = q.grad_t + (size_t)z * N + v;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const float2 g = cadd(X[j], y[j]);
      const float2 tm1 = ts[(z & 1) * N + v + T * j], u = us[(z & 1) * N + v + T * j];
      red_add_cx(grad + T * j, cmulc(g, cfma(tm1, u, u)));
      X[j] = cadd(g, cmulc(g, tm1));
    }
  }
}

// Launches the register kernel of length n, if there is one (*ran = 1).
template <bool BACKWARD>
static int ms_reg_launch(const MsParams &q, cudaStream_t st, int *ran) {
  *ran = 1;
  auto go = [&](auto r2, auto r3) -> int {
    constexpr int R2 = decltype(r2)::value, R3 = decltype(r3)::value;
    auto kern = BACKWARD ? ms_reg_backward_kernel<R2, R3> : ms_reg_march_kernel<R2, R3>;
    constexpr size_t smem = ms_reg_smem<R2, R3>(BACKWARD ? 2 : 1);
    TP_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<q.P, RegFft<R2, R3>::T, smem, st>>>(q);
    return check_cuda(cudaGetLastError(), "multislice register kernel launch");
  };
  using std::integral_constant;
  switch (q.n) {
    case 512: return go(integral_constant<int, 8>{}, integral_constant<int, 4>{});
    case 1024: return go(integral_constant<int, 8>{}, integral_constant<int, 8>{});
    case 2048: return go(integral_constant<int, 16>{}, integral_constant<int, 8>{});
    case 4096: return go(integral_constant<int, 16>{}, integral_constant<int, 16>{});
    default: break;
  }
  *ran = 0;
  return TP_OK;
}

// ------------------------------------------- in-place transforms, other lengths
// The marches at every other n = 2^a 3^b 5^c (fft.cuh's in-place plan), one probe per CTA: a thread keeps the values of its unit of the
// first stage in registers across slices, so that the inverse's last stage, the slice's
// own arithmetic and the next forward transform's first stage need no exchange between
// them; the last forward stage, the product with H - 1 and the first inverse one are a
// single pass.  A slice is 2 (stages - 1) barriers, against two per pass and four more of
// Stockham passes in shared memory: 64 probes, n = 1500 (10 10 15): 9.1 -> 3.3 us per slice
// with the field kept, the adjoint 9.7 -> 3.8 (1000: 6.0 -> 2.6; 243, 32 probes: 4.1 -> 1.9).
template <int R0>
constexpr int kMixThreads = R0 == 5 ? 640 : 512;  // n / R0 at most (625 = 3125 / 5)
template <int R0, bool BACKWARD>
__global__ void __launch_bounds__(kMixThreads<R0>) ms_mix_kernel(const MsParams q, const __grid_constant__ MixPlan pl,
                                                                double gain) {
  extern __shared__ __align__(16) float2 fsm[];
  const int n = q.n, tid = threadIdx.x, nth = blockDim.x, str = pl.str[0];
  float2 *ts = fsm, *us = ts + n, *H = us + (BACKWARD ? n : 0), *tw = H + n, *buf = tw + pl.tw_total;
  const size_t p = blockIdx.x;
  const bool act = tid < str;
  // T - 1 (and u) of a slice into this thread's own slots, issued as soon as those of the
  // slice before are used
  auto stage = [&](int z) {
    if (!act) return;
#pragma unroll
    for (int j = 0; j < R0; ++j) {
      cp_async8(&ts[tid + str * j], &q.trans[(size_t)z * n + tid + str * j]);
      if (BACKWARD) cp_async8(&us[tid + str * j], &q.u_fwd[(p * q.nz + z) * n + tid + str * j]);
    }
    cp_async_commit();
  };
  stage(BACKWARD ? q.L - 1 : 0);
  mix_twiddles(pl, tw, tid, nth);
  __syncthreads();
  __shared__ double red[32];
  gain += cta_sum(mix_twiddle_gain(pl, tw, tid, nth), red);
  const double scale = 1.0 / (n * (1.0 + gain));
  for (int e = tid; e < n; e += nth) {
    const float2 w = ms_h_minus_1(q, mix_frequency(pl, e), scale);
    H[e] = make_float2(w.x, BACKWARD ? -w.y : w.y);
  }
  float2 X[16], y[16];
  float2 *store = !BACKWARD && q.u_store ? q.u_store + p * q.nz * n + tid : nullptr;
  if (act) {
#pragma unroll
    for (int j = 0; j < R0; ++j) {
      X[j] = (BACKWARD ? q.src_exit : q.probes)[p * n + tid + str * j];
      if (store) store[str * j] = X[j];
    }
  }
  __syncthreads();  // twiddles and H are in place
  for (int i = 0; i < q.L; ++i) {
    const int z = BACKWARD ? q.L - 1 - i : i;
    if (act) {
      if (!BACKWARD) {
        cp_async_wait<0>();
#pragma unroll
        for (int j = 0; j < R0; ++j) {
          const float2 t = ts[tid + str * j];
          X[j] = cfma(t, X[j], X[j]);
        }
        if (z + 1 < q.L) stage(z + 1);
      }
#pragma unroll
      for (int j = 0; j < R0; ++j) y[j] = X[j];
      mix_dft<R0>(y, -1.f);
#pragma unroll
      for (int k = 0; k < R0; ++k) buf[mix_pad(tid + str * k)] = k ? cmul(y[k], tw[tid + str * k]) : y[0];
    }
    __syncthreads();
    for (int g = 1; g + 1 < pl.stages; ++g) {
      mix_run<R0, 0>(pl, g, n, buf, tw, H, tid, nth);
      __syncthreads();
    }
    mix_run<R0, 2>(pl, pl.stages - 1, n, buf, tw, H, tid, nth);
    __syncthreads();
    for (int g = pl.stages - 2; g > 0; --g) {
      mix_run<R0, 1>(pl, g, n, buf, tw, H, tid, nth);
      __syncthreads();
    }
    if (!act) continue;
#pragma unroll
    for (int k = 0; k < R0; ++k) {
      const float2 w = buf[mix_pad(tid + str * k)];
      y[k] = k ? cmulc(w, tw[tid + str * k]) : w;
    }
    mix_dft<R0>(y, 1.f);
    if (!BACKWARD) {
      if (store) store += n;
#pragma unroll
      for (int j = 0; j < R0; ++j) {
        X[j] = cadd(X[j], y[j]);
        if (store) __stcs(&store[str * j], X[j]);
      }
    } else {
      cp_async_wait<0>();
      float2 *grad = q.grad_t + (size_t)z * n + tid;
#pragma unroll
      for (int j = 0; j < R0; ++j) {
        const float2 g = cadd(X[j], y[j]);
        const float2 tm1 = ts[tid + str * j], u = us[tid + str * j];
        red_add_cx(grad + str * j, cmulc(g, cfma(tm1, u, u)));
        X[j] = cadd(g, cmulc(g, tm1));
      }
      if (z > 0) stage(z - 1);
    }
  }
  if (!BACKWARD && act && q.exit_out) {
#pragma unroll
    for (int j = 0; j < R0; ++j) q.exit_out[p * n + tid + str * j] = X[j];
  }
}

// Launches the march of length n (which has a plan).
template <bool BACKWARD>
static int ms_launch(const MsParams &q, cudaStream_t st) {
  int ran = 0;
  const int rc = ms_reg_launch<BACKWARD>(q, st, &ran);
  if (rc != TP_OK || ran) return rc;
  const MixPlan pl = make_mix_plan(q.n);
  auto go = [&](auto r0) -> int {
    constexpr int R0 = decltype(r0)::value;
    auto kern = ms_mix_kernel<R0, BACKWARD>;
    const int threads = pl.threads < kMixThreads<R0> ? pl.threads : kMixThreads<R0>;
    const size_t smem = (size_t)((BACKWARD ? 3 : 2) * q.n + pl.tw_total + mix_pad(q.n) + 1) * sizeof(float2);
    TP_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<q.P, threads, smem, st>>>(q, pl, mix_dft_gain(pl));
    return check_cuda(cudaGetLastError(), "multislice in-place kernel launch");
  };
  using std::integral_constant;
  switch (pl.radix[0]) {
    case 16: return go(integral_constant<int, 16>{});
    case 15: return go(integral_constant<int, 15>{});
    case 12: return go(integral_constant<int, 12>{});
    case 10: return go(integral_constant<int, 10>{});
    case 9: return go(integral_constant<int, 9>{});
    case 8: return go(integral_constant<int, 8>{});
    case 6: return go(integral_constant<int, 6>{});
    case 5: return go(integral_constant<int, 5>{});
    case 4: return go(integral_constant<int, 4>{});
    case 3: return go(integral_constant<int, 3>{});
    case 2: return go(integral_constant<int, 2>{});
    default: return set_error(TP_ERR_UNSUPPORTED, "multislice length %d has no plan", q.n);
  }
}

static size_t fft_smem(int n, int rows, int extra) { return (size_t)(extra * n + 2 * rows * n) * sizeof(float2); }

int ms_transmission_launch(int n_total, int nz, double k, double dz, double nmr, double nmi, const void *field,
                           int dtype, float2 *trans, cudaStream_t st) {
  MsParams q{};
  q.n = n_total;
  q.nz = nz;
  q.L = nz - 1;
  q.k = k;
  q.dz = dz;
  q.nmr = nmr;
  q.nmi = nmi;
  q.field = field;
  q.dtype = dtype;
  ms_transmission_kernel<<<592, 256, 0, st>>>(q, trans);
  return check_cuda(cudaGetLastError(), "ms_transmission_kernel launch");
}

static int fft_launch_setup(const void *kern, size_t smem) {
  return check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                    "cudaFuncSetAttribute(fft)");
}

}  // namespace tp

using namespace tp;

static int fft_plan_or_error(int n, FftPlan *pl) {
  *pl = make_fft_plan(n);
  if (pl->npass == 0)
    return set_error(TP_ERR_UNSUPPORTED, "FFT length %d unsupported (need 2^a 3^b 5^c <= %d)", n, kFftMaxN);
  return TP_OK;
}

extern "C" int tp_fft1d(int32_t n, int32_t batch, const void *in, void *out, int32_t inverse, tp_stream_t stream) {
  FftPlan pl;
  int rc = fft_plan_or_error(n, &pl);
  if (rc) return rc;
  if (in == nullptr || out == nullptr || batch < 1) return set_error(TP_ERR_INVALID, "bad tp_fft1d arguments");
  const int rows = fft_rows_per_cta(n);
  const size_t smem = fft_smem(n, rows, 1);
  rc = fft_launch_setup((const void *)fft1d_kernel, smem);
  if (rc) return rc;
  fft1d_kernel<<<(batch + rows - 1) / rows, kFftThreads, smem, reinterpret_cast<cudaStream_t>(stream)>>>(
      pl, batch, static_cast<const float2 *>(in), static_cast<float2 *>(out), inverse, rows);
  return check_cuda(cudaGetLastError(), "fft1d_kernel launch");
}

extern "C" int tp_farfield_intensity(int32_t n, int32_t batch, const void *exit_waves, float *intensity,
                                     tp_stream_t stream) {
  FftPlan pl;
  int rc = fft_plan_or_error(n, &pl);
  if (rc) return rc;
  if (exit_waves == nullptr || intensity == nullptr || batch < 1) return set_error(TP_ERR_INVALID, "bad farfield args");
  const int rows = fft_rows_per_cta(n);
  const size_t smem = fft_smem(n, rows, 1);
  rc = fft_launch_setup((const void *)farfield_kernel, smem);
  if (rc) return rc;
  farfield_kernel<<<(batch + rows - 1) / rows, kFftThreads, smem, reinterpret_cast<cudaStream_t>(stream)>>>(
      pl, batch, static_cast<const float2 *>(exit_waves), intensity, rows);
  return check_cuda(cudaGetLastError(), "farfield_kernel launch");
}

extern "C" int tp_amplitude_residual(int32_t n, int32_t batch, const void *exit_waves, const float *amplitude,
                                     void *grad_out, double *loss_out, tp_stream_t stream) {
  FftPlan pl;
  int rc = fft_plan_or_error(n, &pl);
  if (rc) return rc;
  if (!exit_waves || !amplitude || !grad_out || !loss_out || batch < 1)
    return set_error(TP_ERR_INVALID, "bad amplitude-residual args");
  const int rows = fft_rows_per_cta(n);
  const size_t smem = fft_smem(n, rows, 1);
  rc = fft_launch_setup((const void *)amp_residual_kernel, smem);
  if (rc) return rc;
  amp_residual_kernel<<<(batch + rows - 1) / rows, kFftThreads, smem, reinterpret_cast<cudaStream_t>(stream)>>>(
      pl, batch, static_cast<const float2 *>(exit_waves), amplitude, static_cast<float2 *>(grad_out), loss_out, rows);
  return check_cuda(cudaGetLastError(), "amp_residual_kernel launch");
}

static int ms_params(const tp_ms2d_op *op, MsParams *q) {
  if (op == nullptr) return set_error(TP_ERR_INVALID, "op is NULL");
  if (op->nz < 2) return set_error(TP_ERR_INVALID, "nz=%d must be >= 2", op->nz);
  *q = MsParams{};
  q->n = op->n;
  q->nz = op->nz;
  q->L = op->nz - 1;
  q->k = op->k;
  q->dx = op->dx;
  q->dz = op->dz;
  q->nmr = op->n_medium[0];
  q->nmi = op->n_medium[1];
  return TP_OK;
}

extern "C" int tp_ms2d_transmission(const tp_ms2d_op *op, const void *n_field, int32_t n_dtype, void *trans,
                                    tp_stream_t stream) {
  MsParams q;
  int rc = ms_params(op, &q);
  if (rc) return rc;
  if (!n_field || !trans) return set_error(TP_ERR_INVALID, "n_field/trans is NULL");
  return ms_transmission_launch(q.n, q.nz, q.k, q.dz, q.nmr, q.nmi, n_field, n_dtype, static_cast<float2 *>(trans),
                                reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int tp_ms2d_march(const tp_ms2d_op *op, const void *trans, const void *probes, int32_t num_probes,
                             void *u_store, void *exit_out, tp_stream_t stream) {
  MsParams q;
  int rc = ms_params(op, &q);
  if (rc) return rc;
  FftPlan pl;
  rc = fft_plan_or_error(op->n, &pl);
  if (rc) return rc;
  if (!trans || !probes || num_probes < 1) return set_error(TP_ERR_INVALID, "bad ms march args");
  q.P = num_probes;
  q.trans = static_cast<const float2 *>(trans);
  q.probes = static_cast<const float2 *>(probes);
  q.u_store = static_cast<float2 *>(u_store);
  q.exit_out = static_cast<float2 *>(exit_out);
  return ms_launch<false>(q, reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int tp_ms2d_backward(const tp_ms2d_op *op, const void *trans, const void *u_fwd, const void *src_exit,
                                int32_t num_probes, void *grad_t, tp_stream_t stream) {
  MsParams q;
  int rc = ms_params(op, &q);
  if (rc) return rc;
  FftPlan pl;
  rc = fft_plan_or_error(op->n, &pl);
  if (rc) return rc;
  if (!trans || !u_fwd || !src_exit || !grad_t || num_probes < 1) return set_error(TP_ERR_INVALID, "bad ms backward args");
  q.P = num_probes;
  q.trans = static_cast<const float2 *>(trans);
  q.u_fwd = static_cast<const float2 *>(u_fwd);
  q.src_exit = static_cast<const float2 *>(src_exit);
  q.grad_t = static_cast<float2 *>(grad_t);
  return ms_launch<true>(q, reinterpret_cast<cudaStream_t>(stream));
}
