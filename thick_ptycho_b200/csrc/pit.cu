// Parallel-in-time (PiT) space-time solve of the 2D paraxial march
// (forward_model/pwe/solvers/full_pint.py:71-275 with
// solvers/utils/_pint_utils.py:27-205).
//
// The L = nz - 1 Crank-Nicolson steps form one block-bidiagonal system
//   M u = b,  M = diag(A - C_j) - subdiag(B + C_j),  b = [B u_0, 0, ..., 0]
// (the full-system form: the probe enters through B alone).  It is solved by
// restarted GMRES right-preconditioned with the alpha-circulant
// R = Gamma^-1 F blockdiag((A - w_j B)^-1) F* Gamma: Gamma = diag(alpha^{j/L}),
// F the unitary DFT along z, w_j = alpha^{1/L} e^{2 pi i j/L}, and A, B the
// free-space step matrices (the reference's solver never updates them with C).
//
// B200 mapping: every probe's GMRES runs at once (batched Arnoldi); the
// space-time matvec is one stencil kernel; the z-DFT of arbitrary length L is
// Bluestein's chirp-z on the shared-memory FFT (length M, a power of two
// >= 2L - 1); the L shifted tridiagonal block solves are one thread per
// (probe, frequency) on fp64-built LU factors; the Gram-Schmidt inner
// products (classical, twice) and norms accumulate in fp64.  The host loop
// (Givens rotations, least squares) runs in double complex on the CPU; each
// Arnoldi step reads back (j + 2) numbers per probe.
//
// The Krylov form is flexible GMRES: the preconditioned vectors z_j = R v_j
// are kept and u = u_0 + Z s is built from them.  In exact arithmetic this is
// the reference's right-preconditioned GMRES (u = R y); in fp32 it keeps the
// solution consistent with the Arnoldi relation M Z = V H, whereas forming
// R y at the end adds R's rounding (the z-DFTs and block solves) to the
// residual: at N = 256, L = 127 that floor (~7e-5 ||b||) sat above the
// reference's 1e-5 ||b|| tolerance and the restarts never met it.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <complex>
#include <vector>

#include "fft.cuh"
#include "tp_errors.h"
#include "tpcuda.h"

namespace tp {

constexpr int kPitThreads = 256;
constexpr int kPitMaxRestart = 64;
constexpr int kPitDotGroup = 8;  // basis vectors per inner-product launch

// A tridiagonal K (fp32 copies for the stencils): interior values, the two
// corner diagonals, and one special entry on each off-diagonal (K's at
// K[N-1, N-2] and K[0, 1]; its conjugate transpose's at K^H[1, 0] and
// K^H[N-2, N-1]).
struct PitK {
  int N;
  float2 off, diag, d0, dn;
  int sub_i, sup_i;
  float2 sub_v, sup_v;
  __device__ __forceinline__ float2 sub(int i) const { return i == sub_i ? sub_v : off; }  // K[i, i-1]
  __device__ __forceinline__ float2 sup(int i) const { return i == sup_i ? sup_v : off; }  // K[i, i+1]
  __device__ __forceinline__ float2 dia(int i) const { return i == 0 ? d0 : (i == N - 1 ? dn : diag); }
};
struct PitKd {  // the same in fp64 (block factorisation)
  int N;
  double2 off, diag, d0, dn, k01, knm;
  __device__ __forceinline__ double2 sub(int i) const { return i == N - 1 ? knm : off; }
  __device__ __forceinline__ double2 sup(int i) const { return i == 0 ? k01 : off; }
  __device__ __forceinline__ double2 dia(int i) const { return i == 0 ? d0 : (i == N - 1 ? dn : diag); }
};

// (K v)_i of slice v (length N).
__device__ __forceinline__ float2 pit_kv(const PitK &K, const float2 *v, int i) {
  float2 r = cmul(K.dia(i), v[i]);
  if (i > 0) r = cfma(K.sub(i), v[i - 1], r);
  if (i < K.N - 1) r = cfma(K.sup(i), v[i + 1], r);
  return r;
}

// ------------------------------------------------------------------ object
struct PitObj {
  int N, nz, L, n_obj, empty_px, exact, is_delta, dtype;
  int flip_conj;  // 1: C'[j] = conj(C[L-1-j]) (the reference's adjoint system)
  double k, dz;
  const void *n;
};

__device__ __forceinline__ double2 pit_coef(const PitObj &o, double2 v) {
  const double2 d = o.is_delta ? v : z2(v.x - 1.0, v.y);
  if (!o.exact) return z2(o.k * d.y, -o.k * d.x);      // (k/i) (n - 1)
  const double2 w = zadd(zscale(d, 2.0), zmul(d, d));  // n^2 - 1
  return z2(0.5 * o.k * w.y, -0.5 * o.k * w.x);        // (k/2i) (n^2 - 1)
}

// C[j][i] = (dz/2) * (coef(n[r, j]) + coef(n[r, j+1])) / 2, r = i - empty_px
// (base_simulation_space.py:315-383), slice-major (L, N); with flip_conj the
// z-flipped conjugate the reference's adjoint mode builds (full_pint.py:154-157).
__global__ void pit_object_kernel(const PitObj o, float2 *__restrict__ C) {
  const size_t total = (size_t)o.L * o.N;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
    const int jo = (int)(e / o.N), i = (int)(e % o.N);
    const int j = o.flip_conj ? o.L - 1 - jo : jo;
    const int r = i - o.empty_px;
    double2 c = z2(0.0, 0.0);
    if (r >= 0 && r < o.n_obj) {
      auto ld = [&](int col) {
        const size_t idx = (size_t)r * o.nz + col;
        if (o.dtype == TP_C128) return static_cast<const double2 *>(o.n)[idx];
        const float2 v = static_cast<const float2 *>(o.n)[idx];
        return z2(v.x, v.y);
      };
      c = zscale(zadd(pit_coef(o, ld(j)), pit_coef(o, ld(j + 1))), 0.25 * o.dz);
    }
    C[e] = to_f2(o.flip_conj ? zconj(c) : c);
  }
}

// ------------------------------------------------------------------ matvec
// out = M v for the active probes: slice j gets
// (A - C_j) v_j - (B + C_j) v_{j-1}, A = I - K, B = I + K (_pint_utils.py:27-54;
// the adjoint system passes K^H and the flipped conjugate C).
__global__ void pit_matvec_kernel(const PitK K, int L, int P, const float2 *__restrict__ C,
                                  const float2 *__restrict__ v, float2 *__restrict__ out, const int *active) {
  const int N = K.N;
  const size_t per = (size_t)L * N, total = per * P;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
    const int p = (int)(e / per);
    if (active != nullptr && !active[p]) continue;
    const size_t rem = e - (size_t)p * per;
    const int j = (int)(rem / N), i = (int)(rem % N);
    const float2 *vs = v + (size_t)p * per + (size_t)j * N;
    const float2 c = C[(size_t)j * N + i];
    const float2 x = vs[i];
    float2 r = csub(csub(x, pit_kv(K, vs, i)), cmul(c, x));
    if (j > 0) {
      const float2 *ws = vs - N;
      const float2 y = ws[i];
      r = csub(r, cadd(cadd(y, pit_kv(K, ws, i)), cmul(c, y)));
    }
    out[e] = r;
  }
}

// b[p] = [B u_0 + rhs_0, rhs_1, ...]: u_0 = probes[p] (or zero), rhs (P, L, N) or zero.
__global__ void pit_rhs_kernel(const PitK K, int L, int P, const float2 *__restrict__ probes,
                               const float2 *__restrict__ rhs, float2 *__restrict__ b) {
  const int N = K.N;
  const size_t per = (size_t)L * N, total = per * P;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
    const int p = (int)(e / per);
    const size_t rem = e - (size_t)p * per;
    float2 r = rhs ? rhs[e] : make_float2(0.f, 0.f);
    if (rem < (size_t)N && probes != nullptr) {
      const int i = (int)rem;
      const float2 *u0 = probes + (size_t)p * N;
      r = cadd(r, cadd(u0[i], pit_kv(K, u0, i)));
    }
    b[e] = r;
  }
}

// ------------------------------------------------------------ preconditioner
// Tables: gamma_j = alpha^{j/L}; chirp c_n = exp(-i pi n^2 / L) (n^2 taken
// mod 2L in integers so the fp64 angle stays small); the Bluestein kernel
// b_m = conj(c_m) for |m| < L wrapped into [0, M); twiddles of length M.
__global__ void pit_tables_kernel(int L, int M, double alpha, float *gamma, float2 *chirp, float2 *bker, float2 *tw) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
  for (int j = tid; j < L; j += nth) {
    gamma[j] = (float)pow(alpha, (double)j / (double)L);
    const long long m = ((long long)j * j) % (2LL * L);
    double s, c;
    sincospi(-(double)m / (double)L, &s, &c);
    chirp[j] = make_float2((float)c, (float)s);
  }
  for (int m = tid; m < M; m += nth) {
    int n = -1;
    if (m < L) n = m;
    else if (m > M - L) n = M - m;
    float2 v = make_float2(0.f, 0.f);
    if (n >= 0) {
      const long long q = ((long long)n * n) % (2LL * L);
      double s, c;
      sincospi((double)q / (double)L, &s, &c);  // conj(c_n)
      v = make_float2((float)c, (float)s);
    }
    bker[m] = v;
    double s, c;
    sincospi(-2.0 * (double)m / (double)M, &s, &c);
    tw[m] = make_float2((float)c, (float)s);
  }
}

// Unitary DFT along z by Bluestein's chirp-z, cpc columns per CTA; both domains are
// slice-major (P, L, N).
//   INV (into the block domain): x_j = gamma_j v[p][j][i],
//     out Xh[p][k][i] = (1/sqrt L) sum_j x_j e^{+2 pi i jk/L}
//   !INV (back):  x_k = Xh[p][k][i],
//     out[p][j][i] = (1/sqrt L) sum_k x_k e^{-2 pi i jk/L} / gamma_j
// The inverse direction is conj(DFT(conj x)).  Grid (ceil(N/cpc), P).  Transform
// lengths below 128 on the shared-memory passes.
template <bool INV>
__global__ void __launch_bounds__(kPitThreads) pit_zdft_kernel(const FftPlan pl, int N, int L, int cpc,
                                                               const float2 *__restrict__ in, float2 *__restrict__ out,
                                                               const float *__restrict__ gamma,
                                                               const float2 *__restrict__ chirp,
                                                               const float2 *__restrict__ bhat,
                                                               const float2 *__restrict__ twg, const int *active) {
  extern __shared__ __align__(16) float2 zsm[];
  const int M = pl.n, p = blockIdx.y, i0 = blockIdx.x * cpc;
  if (active != nullptr && !active[p]) return;
  float2 *tw = zsm, *a = tw + M, *b = a + cpc * M;
  load_twiddles(tw, twg, M);
  const size_t base = (size_t)p * L * N + i0;
  for (int e = threadIdx.x; e < cpc * M; e += blockDim.x) a[e] = make_float2(0.f, 0.f);
  __syncthreads();
  for (int e = threadIdx.x; e < cpc * L; e += blockDim.x) {
    const int q = e % cpc, j = e / cpc;  // coalesced over q
    if (i0 + q >= N) continue;
    float2 v = in[base + (size_t)j * N + q];
    if (INV) v = make_float2(gamma[j] * v.x, -gamma[j] * v.y);
    a[q * M + j] = cmul(v, chirp[j]);
  }
  __syncthreads();
  float2 *F = fft_block(a, b, pl, tw, false, cpc, threadIdx.x, blockDim.x);
  float2 *o = (F == a) ? b : a;
  for (int e = threadIdx.x; e < cpc * M; e += blockDim.x) F[e] = cmul(F[e], bhat[e % M]);
  __syncthreads();
  const float2 *R = fft_block(F, o, pl, tw, true, cpc, threadIdx.x, blockDim.x);
  const float sc = 1.f / ((float)M * sqrtf((float)L));
  for (int e = threadIdx.x; e < cpc * L; e += blockDim.x) {
    const int q = e % cpc, j = e / cpc;
    if (i0 + q >= N) continue;
    const float2 X = cmul(R[q * M + j], chirp[j]);
    const float t = INV ? sc : sc / gamma[j];
    out[base + (size_t)j * N + q] = make_float2(t * X.x, INV ? -t * X.y : t * X.y);
  }
}

// The same for M = 16 R2 R3 in 128 .. 4096 with the transforms in registers: M / 16
// threads per column keep 16 values each; the forward transform leaves the spectrum in
// the order of its last step, where it meets bhat and the inverse starts (the steps of
// the 2D multislice's register transforms, ms2d.cu; R3 = 1: two steps).  Threads run
// over the CTA's columns first, so the loads, the stores and the shared-memory exchanges
// move runs of neighbouring columns.  M = 256, 32 x 256 columns: 40 -> 13 us.
template <int R2, int R3>
struct PitFft {
  static constexpr int M = 16 * R2 * R3, T = M / 16, CPC = kPitThreads / T, M2 = 16 / R2, M3 = 16 / R3;
  static constexpr int S1 = T + R3, S2 = ((R2 * (R3 + 1) + 15) / 16) * 16 + R3;
  static constexpr int BUF = 16 * (S1 > S2 ? S1 : S2);
};
template <int R>
__device__ __forceinline__ void pit_dft(float2 *x, float sign) {
  if constexpr (R > 1) {
    float2 w[16];
#pragma unroll
    for (int i = 0; i < R; ++i) w[i] = x[i];
    if constexpr (R == 2) {
      const float2 t = w[0];
      w[0] = cadd(t, w[1]);
      w[1] = csub(t, w[1]);
    } else {
      dft_reg<R>(w, sign);
    }
#pragma unroll
    for (int i = 0; i < R; ++i) x[i] = w[i];
  }
}

template <bool INV, int R2, int R3>
__global__ void __launch_bounds__(kPitThreads, 2) pit_zdft_reg_kernel(int N, int L, const float2 *__restrict__ in,
                                                                      float2 *__restrict__ out,
                                                                      const float *__restrict__ gamma,
                                                                      const float2 *__restrict__ chirp,
                                                                      const float2 *__restrict__ bhat,
                                                                      const float2 *__restrict__ tw, const int *active) {
  using F = PitFft<R2, R3>;
  constexpr int M = F::M, T = F::T, CPC = F::CPC, S1 = F::S1, S2 = F::S2;
  extern __shared__ __align__(16) float2 zsm[];
  const int p = blockIdx.y, i0 = blockIdx.x * CPC;
  if (active != nullptr && !active[p]) return;
  const int q = threadIdx.x % CPC, v = threadIdx.x / CPC;
  float2 *b0 = zsm + q, *b1 = b0 + F::BUF * CPC;  // slot s of this column: s * CPC
  const size_t base = (size_t)p * L * N + i0 + q;
  const bool col = i0 + q < N;
  float2 x[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const int z = v + T * j;
    x[j] = make_float2(0.f, 0.f);
    if (col && z < L) {
      float2 w = in[base + (size_t)z * N];
      if (INV) {
        const float g = gamma[z];
        w = make_float2(g * w.x, -g * w.y);  // conj(x) c_j
      }
      x[j] = cmul(w, chirp[z]);
    }
  }
  pit_dft<16>(x, -1.f);
#pragma unroll
  for (int k = 0; k < 16; ++k) b0[(k * S1 + v) * CPC] = k ? cmul(x[k], tw[v * k]) : x[0];
  __syncthreads();
#pragma unroll
  for (int m = 0; m < F::M2; ++m) {
    const int u = v + T * m, k1 = u / R3, a = u % R3;
#pragma unroll
    for (int b = 0; b < R2; ++b) x[m * R2 + b] = b0[(k1 * S1 + a + R3 * b) * CPC];
    pit_dft<R2>(x + m * R2, -1.f);
    if constexpr (R3 == 1) {
#pragma unroll
      for (int k = 0; k < R2; ++k) x[m * R2 + k] = cmul(x[m * R2 + k], bhat[k1 + 16 * k]);
      pit_dft<R2>(x + m * R2, 1.f);
    } else {
#pragma unroll
      for (int k = 0; k < R2; ++k)
        b1[(k1 * S2 + k * (R3 + 1) + a) * CPC] = k ? cmul(x[m * R2 + k], tw[16 * a * k]) : x[m * R2];
    }
  }
  if constexpr (R3 > 1) {
    __syncthreads();
#pragma unroll
    for (int m = 0; m < F::M3; ++m) {
      const int u = v + T * m, k1 = u / R2, k2 = u % R2;
      float2 *c = b1 + (k1 * S2 + k2 * (R3 + 1)) * CPC;  // this unit's own slots in both directions
#pragma unroll
      for (int a = 0; a < R3; ++a) x[m * R3 + a] = c[a * CPC];
      pit_dft<R3>(x + m * R3, -1.f);
#pragma unroll
      for (int k = 0; k < R3; ++k) x[m * R3 + k] = cmul(x[m * R3 + k], bhat[k1 + 16 * k2 + 16 * R2 * k]);
      pit_dft<R3>(x + m * R3, 1.f);
#pragma unroll
      for (int a = 0; a < R3; ++a) c[a * CPC] = x[m * R3 + a];
    }
    __syncthreads();
  }
#pragma unroll
  for (int m = 0; m < F::M2; ++m) {
    const int u = v + T * m, k1 = u / R3, a = u % R3;
    if constexpr (R3 > 1) {
#pragma unroll
      for (int k = 0; k < R2; ++k) {
        const float2 w = b1[(k1 * S2 + k * (R3 + 1) + a) * CPC];
        x[m * R2 + k] = k ? cmulc(w, tw[16 * a * k]) : w;
      }
      pit_dft<R2>(x + m * R2, 1.f);
    }
#pragma unroll
    for (int b = 0; b < R2; ++b) b0[(k1 * S1 + a + R3 * b) * CPC] = x[m * R2 + b];  // slots this thread read
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const float2 w = b0[(k * S1 + v) * CPC];
    x[k] = k ? cmulc(w, tw[v * k]) : w;
  }
  pit_dft<16>(x, 1.f);
  const float sc = 1.f / ((float)M * sqrtf((float)L));
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const int z = v + T * j;
    if (!col || z >= L) continue;
    const float2 X = cmul(x[j], chirp[z]);
    const float t = INV ? sc : sc / gamma[z];
    out[base + (size_t)z * N] = make_float2(t * X.x, INV ? -t * X.y : t * X.y);
  }
}

// LU factors of the L blocks (A - w_k B) = (1 - w_k) I - (1 + w_k) K, fp64
// Thomas elimination, stored as float4 (m_i, 1/d_i) at [k][i].
__global__ void pit_factor_kernel(const PitKd K, int L, double alpha_root, float4 *__restrict__ F) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= L) return;
  double s, c;
  sincospi(2.0 * (double)k / (double)L, &s, &c);
  const double2 w = z2(alpha_root * c, alpha_root * s);
  const double2 omw = z2(1.0 - w.x, -w.y), opw = z2(1.0 + w.x, w.y);
  auto dval = [&](int i) { return zsub(omw, zmul(opw, K.dia(i))); };
  double2 d = dval(0);
  double2 dinv = zinv(d);
  F += (size_t)k * K.N;
  F[0] = make_float4(0.f, 0.f, (float)dinv.x, (float)dinv.y);
  for (int i = 1; i < K.N; ++i) {
    const double2 a = zneg(zmul(opw, K.sub(i)));          // row i, column i-1
    const double2 cprev = zneg(zmul(opw, K.sup(i - 1)));  // row i-1, column i
    const double2 m = zmul(a, dinv);
    d = zsub(dval(i), zmul(m, cprev));
    dinv = zinv(d);
    F[i] = make_float4((float)m.x, (float)m.y, (float)dinv.x, (float)dinv.y);
  }
}

// Block solves in place on Xh (P, L, N): warp (p, k) solves along i, kPitRows rows per
// lane at a time.  Both sweeps are first-order recurrences y_i = x_i + c_i y_{i-1} (c =
// -m forward; c_i = -sup_i / d_i on y / d backward): a lane runs its rows from zero and
// the products of their c, the lanes' (product, last y) pairs are combined by a warp
// scan, and each row adds its product times what enters its lane.  One thread per block
// instead runs N dependent rows twice: N = 256, 4064 blocks: 42 -> 14 us.
constexpr int kPitRows = 8;
struct PitAffine {
  float2 a, b;  // y -> a y + b
};
// What enters this lane: the composition of all earlier lanes' maps applied to `carry`
// (DOWN: of all later lanes'); carry becomes the value behind the last one.
template <bool DOWN>
__device__ __forceinline__ float2 pit_enter(PitAffine f, float2 &carry) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int s = 1; s < 32; s <<= 1) {
    const float2 a = DOWN ? shfl_down2(f.a, s) : shfl_up2(f.a, s), b = DOWN ? shfl_down2(f.b, s) : shfl_up2(f.b, s);
    if (DOWN ? lane + s < 32 : lane >= s) {
      f.b = cfma(f.a, b, f.b);
      f.a = cmul(f.a, a);
    }
  }
  const float2 y = cfma(f.a, carry, f.b);
  const float2 prev = DOWN ? shfl_down2(y, 1) : shfl_up2(y, 1);
  const float2 in = (DOWN ? lane == 31 : lane == 0) ? carry : prev;
  const int last = DOWN ? 0 : 31;
  carry = make_float2(__shfl_sync(0xffffffffu, y.x, last), __shfl_sync(0xffffffffu, y.y, last));
  return in;
}
__global__ void __launch_bounds__(256) pit_block_solve_kernel(const PitK K, int L, int P, double alpha_root,
                                                              const float4 *__restrict__ F, float2 *__restrict__ Xh,
                                                              const int *active) {
  const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (t >= L * P) return;
  const int p = t / L, k = t % L;
  if (active != nullptr && !active[p]) return;
  const int N = K.N;
  double s, c;
  sincospi(2.0 * (double)k / (double)L, &s, &c);
  const float2 mopw = make_float2((float)-(1.0 + alpha_root * c), (float)-(alpha_root * s));
  float2 *x = Xh + (size_t)t * N;
  const float4 *f = F + (size_t)k * N;
  constexpr int R = kPitRows, TILE = 32 * R;
  const float2 zero = make_float2(0.f, 0.f);
  const int tiles = (N + TILE - 1) / TILE;
  float2 y[R], a[R], di[R], carry = zero;
  for (int n = 0; n < tiles; ++n) {
    const int i0 = n * TILE + lane * R;
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const bool in = i0 + j < N;
      const float4 v = in ? f[i0 + j] : make_float4(0.f, 0.f, 0.f, 0.f);
      y[j] = in ? x[i0 + j] : zero;
      a[j] = make_float2(-v.x, -v.y);
      di[j] = make_float2(v.z, v.w);
    }
#pragma unroll
    for (int j = 1; j < R; ++j) {
      y[j] = cfma(a[j], y[j - 1], y[j]);
      a[j] = cmul(a[j], a[j - 1]);
    }
    const float2 in = pit_enter<false>({a[R - 1], y[R - 1]}, carry);
#pragma unroll
    for (int j = 0; j < R; ++j) y[j] = cfma(a[j], in, y[j]);
    if (n + 1 < tiles) {  // the last tile stays in registers
#pragma unroll
      for (int j = 0; j < R; ++j) x[i0 + j] = y[j];
    }
  }
  carry = zero;
  for (int n = tiles - 1; n >= 0; --n) {
    const int i0 = n * TILE + lane * R;
    if (n < tiles - 1) {
#pragma unroll
      for (int j = 0; j < R; ++j) {
        const float4 v = f[i0 + j];
        y[j] = x[i0 + j];
        di[j] = make_float2(v.z, v.w);
      }
    }
#pragma unroll
    for (int j = 0; j < R; ++j) {  // y_i / d_i - (c_i / d_i) y_{i+1}, c_i row i's coupling to column i + 1
      const int i = i0 + j;
      a[j] = i < N - 1 ? cmul(cmul(mopw, K.sup(i)), make_float2(-di[j].x, -di[j].y)) : zero;
      y[j] = cmul(y[j], di[j]);
    }
#pragma unroll
    for (int j = R - 2; j >= 0; --j) {
      y[j] = cfma(a[j], y[j + 1], y[j]);
      a[j] = cmul(a[j], a[j + 1]);
    }
    const float2 in = pit_enter<true>({a[0], y[0]}, carry);
#pragma unroll
    for (int j = 0; j < R; ++j)
      if (i0 + j < N) x[i0 + j] = cfma(a[j], in, y[j]);
  }
}

// ------------------------------------------------------------------ Krylov
// dst[r] += the CTA's sums of the first cnt complex accumulators.
__device__ __forceinline__ void pit_reduce_dots(const double (&acc)[2 * kPitDotGroup], int cnt,
                                                double (*red)[2 * kPitDotGroup], double2 *dst) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int r = 0; r < 2 * kPitDotGroup; ++r) {
    if (r >= 2 * cnt) break;
    double v = acc[r];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) red[wid][r] = v;
  }
  __syncthreads();
  if (threadIdx.x < 2 * cnt) {
    double s = 0.0;
    for (int q = 0; q < kPitThreads / 32; ++q) s += red[q][threadIdx.x];
    atomicAdd(reinterpret_cast<double *>(&dst[threadIdx.x >> 1]) + (threadIdx.x & 1), s);
  }
}

// h[p][r0 + r] += <V_{r0+r}[p], w[p]> (fp64) for r < min(kPitDotGroup, nv - r0).
__global__ void __launch_bounds__(kPitThreads) pit_dots_kernel(size_t n, int P, const float2 *__restrict__ V,
                                                               size_t vstride, int r0, int nv,
                                                               const float2 *__restrict__ w, double2 *h, int hld,
                                                               const int *active) {
  const int p = blockIdx.y;
  if (active != nullptr && !active[p]) return;
  __shared__ double red[kPitThreads / 32][2 * kPitDotGroup];
  double acc[2 * kPitDotGroup];
#pragma unroll
  for (int r = 0; r < 2 * kPitDotGroup; ++r) acc[r] = 0.0;
  const int cnt = min(kPitDotGroup, nv - r0);
  const float2 *wp = w + (size_t)p * n;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
    const float2 x = wp[e];
#pragma unroll
    for (int r = 0; r < kPitDotGroup; ++r) {
      if (r < cnt) {
        const float2 v = V[(size_t)(r0 + r) * vstride + (size_t)p * n + e];
        acc[2 * r] += (double)v.x * x.x + (double)v.y * x.y;  // conj(v) x
        acc[2 * r + 1] += (double)v.x * x.y - (double)v.y * x.x;
      }
    }
  }
  pit_reduce_dots(acc, cnt, red, &h[(size_t)p * hld + r0]);
}

// w[p] += sign * sum_{r < nv} coef[p][r] V_r[p]  (coef fp64, per probe); nrm (or
// NULL): nrm[p] += ||w[p]||^2 of the result.
__global__ void __launch_bounds__(kPitThreads) pit_combine_kernel(size_t n, int P, const float2 *__restrict__ V,
                                                                  size_t vstride, int nv,
                                                                  const double2 *__restrict__ coef, int cld,
                                                                  float sign, float2 *__restrict__ w, double *nrm,
                                                                  const int *active) {
  const int p = blockIdx.y;
  if (active != nullptr && !active[p]) return;
  __shared__ double red[kPitThreads / 32];
  double sum = 0.0;
  __shared__ float2 cf[kPitMaxRestart + 1];
  for (int r = threadIdx.x; r < nv; r += blockDim.x) {
    const double2 c = coef[(size_t)p * cld + r];
    cf[r] = make_float2((float)(sign * c.x), (float)(sign * c.y));
  }
  __syncthreads();
  float2 *wp = w + (size_t)p * n;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
    float2 acc = wp[e];
    for (int r = 0; r < nv; ++r) acc = cfma(cf[r], V[(size_t)r * vstride + (size_t)p * n + e], acc);
    wp[e] = acc;
    if (nrm != nullptr) sum += (double)acc.x * acc.x + (double)acc.y * acc.y;
  }
  if (nrm == nullptr) return;
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int q = 0; q < kPitThreads / 32; ++q) s += red[q];
    atomicAdd(&nrm[p], s);
  }
}

// The second Gram-Schmidt pass' first half in one reading of the basis (nv <=
// kPitDotGroup): w[p] -= sum_r coef[p][r] V_r[p], then h[p][r] += <V_r[p], w[p]>.
__global__ void __launch_bounds__(kPitThreads) pit_combine_dots_kernel(size_t n, const float2 *__restrict__ V,
                                                                       size_t vstride, int nv,
                                                                       const double2 *__restrict__ coef, int cld,
                                                                       float2 *__restrict__ w, double2 *h,
                                                                       const int *active) {
  const int p = blockIdx.y;
  if (active != nullptr && !active[p]) return;
  __shared__ double red[kPitThreads / 32][2 * kPitDotGroup];
  float2 cf[kPitDotGroup];
  double acc[2 * kPitDotGroup];
#pragma unroll
  for (int r = 0; r < kPitDotGroup; ++r) {
    acc[2 * r] = acc[2 * r + 1] = 0.0;
    const double2 c = r < nv ? coef[(size_t)p * cld + r] : z2(0.0, 0.0);
    cf[r] = make_float2((float)-c.x, (float)-c.y);
  }
  float2 *wp = w + (size_t)p * n;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
    float2 v[kPitDotGroup], x = wp[e];
#pragma unroll
    for (int r = 0; r < kPitDotGroup; ++r)
      if (r < nv) v[r] = V[(size_t)r * vstride + (size_t)p * n + e];
#pragma unroll
    for (int r = 0; r < kPitDotGroup; ++r)
      if (r < nv) x = cfma(cf[r], v[r], x);
    wp[e] = x;
#pragma unroll
    for (int r = 0; r < kPitDotGroup; ++r) {
      if (r < nv) {
        acc[2 * r] += (double)v[r].x * x.x + (double)v[r].y * x.y;
        acc[2 * r + 1] += (double)v[r].x * x.y - (double)v[r].y * x.x;
      }
    }
  }
  pit_reduce_dots(acc, nv, red, &h[(size_t)p * cld]);
}

// nrm[p] += ||x[p]||^2 (fp64)
__global__ void __launch_bounds__(kPitThreads) pit_norm_kernel(size_t n, int P, const float2 *__restrict__ x,
                                                               double *nrm, const int *active) {
  const int p = blockIdx.y;
  if (active != nullptr && !active[p]) return;
  __shared__ double red[kPitThreads / 32];
  double acc = 0.0;
  const float2 *xp = x + (size_t)p * n;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
    const float2 v = xp[e];
    acc += (double)v.x * v.x + (double)v.y * v.y;
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int q = 0; q < kPitThreads / 32; ++q) s += red[q];
    atomicAdd(&nrm[p], s);
  }
}

// out[p] = s[p] * x[p]   |   out[p] = x[p] - y[p] (s == NULL)
__global__ void pit_scale_kernel(size_t n, int P, const float2 *__restrict__ x, const float2 *__restrict__ y,
                                 const double *s, float2 *__restrict__ out, const int *active) {
  const size_t total = n * P;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
    const int p = (int)(e / n);
    if (active != nullptr && !active[p]) continue;
    if (s != nullptr) {
      const float f = (float)s[p];
      out[e] = make_float2(f * x[e].x, f * x[e].y);
    } else {
      out[e] = csub(x[e], y[e]);
    }
  }
}

// ------------------------------------------------------------------ host
struct PitWork {
  float2 *V, *Z, *w, *xh, *b, *C, *chirp, *bker, *bhat, *tw;
  float4 *F;
  float *gamma;
  // the two passes' inner products (P x hld each) and the norms, back to back
  double2 *h, *h2;
  double *nrm, *s;
  int *active;
  size_t bytes;
};

static size_t pit_a256(size_t b) { return (b + 255) & ~(size_t)255; }

static int pit_fft_len(int L) {
  int M = 4;
  while (M < 2 * L - 1) M *= 2;
  return M;
}

static PitWork pit_layout(char *base, int N, int L, int P, int m) {
  PitWork w{};
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char *p = base ? base + off : nullptr;
    off += pit_a256(bytes);
    return p;
  };
  const size_t n = (size_t)N * L, vec = n * P * sizeof(float2);
  const int M = pit_fft_len(L);
  w.V = reinterpret_cast<float2 *>(take(vec * (m + 1)));
  w.Z = reinterpret_cast<float2 *>(take(vec * m));
  w.w = reinterpret_cast<float2 *>(take(vec));
  w.xh = reinterpret_cast<float2 *>(take(vec));
  w.b = reinterpret_cast<float2 *>(take(vec));
  w.C = reinterpret_cast<float2 *>(take(n * sizeof(float2)));
  w.F = reinterpret_cast<float4 *>(take(n * sizeof(float4)));
  w.gamma = reinterpret_cast<float *>(take((size_t)L * sizeof(float)));
  w.chirp = reinterpret_cast<float2 *>(take((size_t)L * sizeof(float2)));
  w.bker = reinterpret_cast<float2 *>(take((size_t)M * sizeof(float2)));
  w.bhat = reinterpret_cast<float2 *>(take((size_t)M * sizeof(float2)));
  w.tw = reinterpret_cast<float2 *>(take((size_t)M * sizeof(float2)));
  const size_t hlen = (size_t)P * (kPitMaxRestart + 1);
  w.h = reinterpret_cast<double2 *>(take(2 * hlen * sizeof(double2) + (size_t)P * sizeof(double)));
  w.h2 = w.h + hlen;
  w.nrm = reinterpret_cast<double *>(w.h + 2 * hlen);
  w.s = reinterpret_cast<double *>(take((size_t)P * sizeof(double)));
  w.active = reinterpret_cast<int *>(take((size_t)P * sizeof(int)));
  w.bytes = off;
  return w;
}

// K of the operator, or its conjugate transpose (conj_t): K^H[i, i-1] =
// conj(K[i-1, i]) and K^H[i, i+1] = conj(K[i+1, i]).
static PitK pit_k(const tp_cn2d_op *op, bool conj_t = false) {
  auto f = [&](const double v[2]) { return make_float2((float)v[0], (float)(conj_t ? -v[1] : v[1])); };
  const int N = op->n;
  if (!conj_t) return PitK{N, f(op->k_off), f(op->k_diag), f(op->k_d0), f(op->k_dn), N - 1, 0, f(op->k_nm), f(op->k_01)};
  return PitK{N, f(op->k_off), f(op->k_diag), f(op->k_d0), f(op->k_dn), 1, N - 2, f(op->k_01), f(op->k_nm)};
}
static PitKd pit_kd(const tp_cn2d_op *op) {
  auto f = [](const double v[2]) { return make_double2(v[0], v[1]); };
  return PitKd{op->n, f(op->k_off), f(op->k_diag), f(op->k_d0), f(op->k_dn), f(op->k_01), f(op->k_nm)};
}

static int pit_grid(size_t total) {
  const size_t g = (total + kPitThreads - 1) / kPitThreads;
  return (int)(g < 4 * 148 ? (g < 1 ? 1 : g) : 4 * 148);
}

// Device-side pieces of one solve: the preconditioner, the space-time matvec
// and the batched Gram-Schmidt kernels, over all probes.
class PitSolver {
 public:
  PitSolver(const tp_cn2d_op *op, int L, int P, const PitWork &w, cudaStream_t st, bool adjoint = false)
      : K_(pit_k(op)), KM_(pit_k(op, adjoint)), kd_(pit_kd(op)), N_(op->n), L_(L), P_(P), n_((size_t)op->n * L),
        w_(w), st_(st) {
    M_ = pit_fft_len(L);
    pl_ = make_fft_plan(M_);
    cpc_ = std::max(1, std::min(16, 4096 / M_));
    zsmem_ = (size_t)(M_ + 2 * cpc_ * M_) * sizeof(float2);
  }

  int setup(double alpha) {
    alpha_root_ = pow(alpha, 1.0 / (double)L_);
    pit_tables_kernel<<<8, 256, 0, st_>>>(L_, M_, alpha, w_.gamma, w_.chirp, w_.bker, w_.tw);
    TP_CHECK_CUDA(cudaGetLastError());
    int rc = tp_fft1d(M_, 1, w_.bker, w_.bhat, 0, reinterpret_cast<tp_stream_t>(st_));
    if (rc) return rc;
    pit_factor_kernel<<<(L_ + 127) / 128, 128, 0, st_>>>(kd_, L_, alpha_root_, w_.F);
    TP_CHECK_CUDA(cudaGetLastError());
    TP_CHECK_CUDA(cudaFuncSetAttribute(pit_zdft_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)zsmem_));
    TP_CHECK_CUDA(cudaFuncSetAttribute(pit_zdft_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)zsmem_));
    return TP_OK;
  }
  template <bool INV, int R2, int R3>
  int zdft_reg(const float2 *in, float2 *out) {
    using F = PitFft<R2, R3>;
    constexpr size_t smem = (size_t)(R3 > 1 ? 2 : 1) * F::BUF * F::CPC * sizeof(float2);
    auto kern = pit_zdft_reg_kernel<INV, R2, R3>;
    TP_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<dim3((N_ + F::CPC - 1) / F::CPC, P_), kPitThreads, smem, st_>>>(N_, L_, in, out, w_.gamma, w_.chirp, w_.bhat,
                                                                          w_.tw, w_.active);
    return check_cuda(cudaGetLastError(), "pit_zdft_reg_kernel launch");
  }
  template <bool INV>
  int zdft(const float2 *in, float2 *out) {
    switch (M_) {
      case 128: return zdft_reg<INV, 8, 1>(in, out);
      case 256: return zdft_reg<INV, 16, 1>(in, out);
      case 512: return zdft_reg<INV, 8, 4>(in, out);
      case 1024: return zdft_reg<INV, 8, 8>(in, out);
      case 2048: return zdft_reg<INV, 16, 8>(in, out);
      case 4096: return zdft_reg<INV, 16, 16>(in, out);
      default: break;
    }
    pit_zdft_kernel<INV><<<dim3((N_ + cpc_ - 1) / cpc_, P_), kPitThreads, zsmem_, st_>>>(
        pl_, N_, L_, cpc_, in, out, w_.gamma, w_.chirp, w_.bhat, w_.tw, w_.active);
    return check_cuda(cudaGetLastError(), "pit_zdft_kernel launch");
  }

  // out = R in (the preconditioner), active probes only.
  int precond(const float2 *in, float2 *out) {
    int rc = zdft<true>(in, w_.xh);
    if (rc) return rc;
    const size_t threads = (size_t)L_ * P_ * 32;
    pit_block_solve_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, st_>>>(K_, L_, P_, alpha_root_, w_.F, w_.xh,
                                                                              w_.active);
    rc = zdft<false>(w_.xh, out);
    if (rc) return rc;
    return check_cuda(cudaGetLastError(), "pit preconditioner launch");
  }
  // out = M in (M of the forward or the reference's adjoint system)
  int matvec(const float2 *in, float2 *out) {
    pit_matvec_kernel<<<pit_grid(n_ * P_), kPitThreads, 0, st_>>>(KM_, L_, P_, w_.C, in, out, w_.active);
    return check_cuda(cudaGetLastError(), "pit matvec launch");
  }
  // out[p] = ||x[p]||^2 on the host
  int norms(const float2 *x, std::vector<double> &out) {
    TP_CHECK_CUDA(cudaMemsetAsync(w_.nrm, 0, P_ * sizeof(double), st_));
    pit_norm_kernel<<<dim3(red_blocks(), P_), kPitThreads, 0, st_>>>(n_, P_, x, w_.nrm, w_.active);
    TP_CHECK_CUDA(cudaGetLastError());
    out.resize(P_);
    TP_CHECK_CUDA(cudaMemcpyAsync(out.data(), w_.nrm, P_ * sizeof(double), cudaMemcpyDeviceToHost, st_));
    TP_CHECK_CUDA(cudaStreamSynchronize(st_));
    return TP_OK;
  }
  // w orthogonalised against V_0..V_{nv-1} by classical Gram-Schmidt, twice: the two
  // passes' products in w_.h and w_.h2 and the remaining norms in w_.nrm, read back
  // together (one host wait per Arnoldi step).
  int orthogonalise(int nv, float2 *w, std::vector<double> &out) {
    const size_t hlen = (size_t)P_ * (kPitMaxRestart + 1), bytes = 2 * hlen * sizeof(double2) + P_ * sizeof(double);
    TP_CHECK_CUDA(cudaMemsetAsync(w_.h, 0, bytes, st_));
    const dim3 grid(red_blocks(), P_);
    auto dots = [&](double2 *h) {
      for (int r0 = 0; r0 < nv; r0 += kPitDotGroup)
        pit_dots_kernel<<<grid, kPitThreads, 0, st_>>>(n_, P_, w_.V, n_ * P_, r0, nv, w, h, kPitMaxRestart + 1, w_.active);
    };
    dots(w_.h);
    if (nv <= kPitDotGroup) {
      pit_combine_dots_kernel<<<grid, kPitThreads, 0, st_>>>(n_, w_.V, n_ * P_, nv, w_.h, kPitMaxRestart + 1, w, w_.h2,
                                                             w_.active);
    } else {
      pit_combine_kernel<<<grid, kPitThreads, 0, st_>>>(n_, P_, w_.V, n_ * P_, nv, w_.h, kPitMaxRestart + 1, -1.f, w,
                                                        nullptr, w_.active);
      dots(w_.h2);
    }
    pit_combine_kernel<<<grid, kPitThreads, 0, st_>>>(n_, P_, w_.V, n_ * P_, nv, w_.h2, kPitMaxRestart + 1, -1.f, w,
                                                      w_.nrm, w_.active);
    TP_CHECK_CUDA(cudaGetLastError());
    out.resize(bytes / sizeof(double));
    TP_CHECK_CUDA(cudaMemcpyAsync(out.data(), w_.h, bytes, cudaMemcpyDeviceToHost, st_));
    TP_CHECK_CUDA(cudaStreamSynchronize(st_));
    return TP_OK;
  }
  // target += sign * sum_r h[p][r] basis_r[p]
  int combine(const float2 *basis, int nv, float sign, float2 *target) {
    pit_combine_kernel<<<dim3(red_blocks(), P_), kPitThreads, 0, st_>>>(n_, P_, basis, n_ * P_, nv, w_.h,
                                                                       kPitMaxRestart + 1, sign, target, nullptr,
                                                                       w_.active);
    return check_cuda(cudaGetLastError(), "pit combine launch");
  }
  int red_blocks() const {
    // enough CTAs for every SM over all probes; more would spend their time on the
    // sums at their ends (dots of 32 probes, 32512 elements: 22 us with 64 per probe)
    const size_t g = (n_ + kPitThreads - 1) / kPitThreads;
    const size_t want = (size_t)std::max(1, std::min(64, (4 * 148 + P_ - 1) / P_));
    return (int)(g < want ? g : want);
  }

  PitK K_;   // the operator's K: right-hand side, preconditioner blocks
  PitK KM_;  // K of the system matrix: K, or K^H in the adjoint mode
  PitKd kd_;
  int N_, L_, P_, M_ = 0, cpc_ = 1;
  size_t n_, zsmem_ = 0;
  double alpha_root_ = 1.0;
  FftPlan pl_{};
  PitWork w_;
  cudaStream_t st_;
};

}  // namespace tp

using namespace tp;

extern "C" size_t tp_pit_workspace_bytes(int32_t n, int32_t nz, int32_t num_probes, int32_t restart) {
  if (n < 2 || nz < 3 || num_probes < 1) return 0;
  const int m = restart > 0 ? restart : 20;
  if (m > kPitMaxRestart) return 0;
  return pit_layout(nullptr, n, nz - 1, num_probes, m).bytes;
}

extern "C" int tp_pit_solve(const tp_cn2d_op *op, const void *n_field, int32_t n_dtype, const tp_pit_args *a,
                            void *workspace, size_t workspace_bytes, tp_stream_t stream) {
  if (op == nullptr || a == nullptr || n_field == nullptr || workspace == nullptr)
    return set_error(TP_ERR_INVALID, "tp_pit_solve: NULL argument");
  const int N = op->n, L = op->nz - 1, P = a->num_probes;
  const int m = a->restart > 0 ? a->restart : 20;
  if (N < 2 || L < 2 || P < 1) return set_error(TP_ERR_INVALID, "tp_pit_solve: N=%d, nz=%d, P=%d", N, op->nz, P);
  if (m > kPitMaxRestart) return set_error(TP_ERR_INVALID, "restart=%d > %d", m, kPitMaxRestart);
  if (2 * L - 1 > kFftMaxN)
    return set_error(TP_ERR_UNSUPPORTED, "PiT needs nz - 1 <= %d (got %d)", (kFftMaxN + 1) / 2, L);
  if (a->u == nullptr) return set_error(TP_ERR_INVALID, "tp_pit_solve: u is required");
  if (op->n_obj + 2 * op->empty_px != N) return set_error(TP_ERR_INVALID, "n_obj + 2 empty_px != n");
  if ((reinterpret_cast<uintptr_t>(workspace) & 255u) != 0)
    return set_error(TP_ERR_INVALID, "workspace must be 256-byte aligned");
  const PitWork w = pit_layout(static_cast<char *>(workspace), N, L, P, m);
  if (workspace_bytes < w.bytes)
    return set_error(TP_ERR_WORKSPACE, "PiT workspace %zu B < %zu B", workspace_bytes, w.bytes);
  const double alpha = a->alpha > 0 ? a->alpha : 1e-2;
  const double rtol = a->rtol > 0 ? a->rtol : 1e-5, atol = a->atol > 0 ? a->atol : 1e-8;
  const int max_cycles = a->max_cycles > 0 ? a->max_cycles : 1000;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const size_t n = (size_t)N * L;

  if (a->mode != TP_MODE_FORWARD && a->mode != TP_MODE_ADJOINT)
    return set_error(TP_ERR_UNSUPPORTED, "tp_pit_solve: mode %d (FORWARD or ADJOINT)", a->mode);
  const bool adjoint = a->mode == TP_MODE_ADJOINT;
  PitSolver S(op, L, P, w, st, adjoint);
  // object contribution (slice-major) and right-hand sides
  PitObj o{N, op->nz, L, op->n_obj, op->empty_px, op->exact_ref_coeff, op->field_is_delta, n_dtype, adjoint ? 1 : 0,
           op->k, op->dz, n_field};
  pit_object_kernel<<<pit_grid(n), kPitThreads, 0, st>>>(o, w.C);
  pit_rhs_kernel<<<pit_grid(n * P), kPitThreads, 0, st>>>(S.K_, L, P, static_cast<const float2 *>(a->probes),
                                                           static_cast<const float2 *>(a->rhs), w.b);
  TP_CHECK_CUDA(cudaGetLastError());
  int rc = S.setup(alpha);
  if (rc) return rc;

  float2 *u = static_cast<float2 *>(a->u);
  std::vector<int> active(P, 1), iters(P, 0);
  std::vector<double> tol(P), bn, rn;
  TP_CHECK_CUDA(cudaMemcpyAsync(w.active, active.data(), P * sizeof(int), cudaMemcpyHostToDevice, st));
  rc = S.norms(w.b, bn);
  if (rc) return rc;
  for (int p = 0; p < P; ++p) tol[p] = std::fmax(atol, rtol * std::sqrt(bn[p]));

  using cd = std::complex<double>;
  std::vector<cd> H((size_t)P * (m + 1) * m), cs((size_t)P * m), sn((size_t)P * m), g((size_t)P * (m + 1));
  std::vector<double2> hh((size_t)P * (kPitMaxRestart + 1));
  std::vector<double> back;
  std::vector<int> inner(P), kdim(P);
  auto Hat = [&](int p, int r, int c) -> cd & { return H[((size_t)p * (m + 1) + r) * m + c]; };

  for (int cyc = 0; cyc < max_cycles; ++cyc) {
    // r = b - M u for every probe still running
    rc = S.matvec(u, w.w);
    if (rc) return rc;
    pit_scale_kernel<<<pit_grid(n * P), kPitThreads, 0, st>>>(n, P, w.b, w.w, nullptr, w.w, w.active);
    rc = S.norms(w.w, rn);
    if (rc) return rc;
    bool any = false;
    for (int p = 0; p < P; ++p) {
      if (!active[p]) continue;
      if (std::sqrt(rn[p]) <= tol[p]) active[p] = 0;
      else any = true;
    }
    if (!any) break;
    TP_CHECK_CUDA(cudaMemcpyAsync(w.active, active.data(), P * sizeof(int), cudaMemcpyHostToDevice, st));
    std::vector<double> sc(P, 0.0);
    for (int p = 0; p < P; ++p) {
      inner[p] = active[p];
      kdim[p] = 0;
      std::fill(g.begin() + (size_t)p * (m + 1), g.begin() + (size_t)(p + 1) * (m + 1), cd(0.0));
      if (active[p]) {
        const double beta = std::sqrt(rn[p]);
        g[(size_t)p * (m + 1)] = beta;
        sc[p] = 1.0 / beta;
      }
    }
    TP_CHECK_CUDA(cudaMemcpyAsync(w.s, sc.data(), P * sizeof(double), cudaMemcpyHostToDevice, st));
    pit_scale_kernel<<<pit_grid(n * P), kPitThreads, 0, st>>>(n, P, w.w, nullptr, w.s, w.V, w.active);
    for (int j = 0; j < m; ++j) {
      float2 *Vj = w.V + (size_t)j * n * P, *Zj = w.Z + (size_t)j * n * P;
      rc = S.precond(Vj, Zj);
      if (rc) return rc;
      rc = S.matvec(Zj, w.w);
      if (rc) return rc;
      rc = S.orthogonalise(j + 1, w.w, back);
      if (rc) return rc;
      const size_t hlen = (size_t)P * (kPitMaxRestart + 1);
      const cd *h1 = reinterpret_cast<const cd *>(back.data()), *h2 = h1 + hlen;
      const double *nrm = back.data() + 4 * hlen;
      bool cont = false;
      for (int p = 0; p < P; ++p) {
        sc[p] = 0.0;
        if (!inner[p]) continue;
        for (int r = 0; r <= j; ++r) {
          const size_t at = (size_t)p * (kPitMaxRestart + 1) + r;
          Hat(p, r, j) = h1[at] + h2[at];
        }
        const double eta = std::sqrt(nrm[p]);
        Hat(p, j + 1, j) = eta;
        cd *csp = &cs[(size_t)p * m], *snp = &sn[(size_t)p * m], *gp = &g[(size_t)p * (m + 1)];
        for (int r = 0; r < j; ++r) {  // previous rotations
          const cd h0 = Hat(p, r, j), h1 = Hat(p, r + 1, j);
          Hat(p, r, j) = std::conj(csp[r]) * h0 + std::conj(snp[r]) * h1;
          Hat(p, r + 1, j) = -snp[r] * h0 + csp[r] * h1;
        }
        const cd a0 = Hat(p, j, j), a1 = Hat(p, j + 1, j);
        const double den = std::sqrt(std::norm(a0) + std::norm(a1));
        csp[j] = den > 0 ? a0 / den : cd(1.0);
        snp[j] = den > 0 ? a1 / den : cd(0.0);
        Hat(p, j, j) = den;
        Hat(p, j + 1, j) = 0.0;
        gp[j + 1] = -snp[j] * gp[j];
        gp[j] = std::conj(csp[j]) * gp[j];
        iters[p] += 1;
        kdim[p] = j + 1;
        if (std::abs(gp[j + 1]) <= tol[p] || eta == 0.0 || j == m - 1) {
          inner[p] = 0;
        } else {
          sc[p] = 1.0 / eta;
          cont = true;
        }
      }
      if (!cont) break;
      // V_{j+1} = w / eta for the probes that continue
      TP_CHECK_CUDA(cudaMemcpyAsync(w.active, inner.data(), P * sizeof(int), cudaMemcpyHostToDevice, st));
      TP_CHECK_CUDA(cudaMemcpyAsync(w.s, sc.data(), P * sizeof(double), cudaMemcpyHostToDevice, st));
      pit_scale_kernel<<<pit_grid(n * P), kPitThreads, 0, st>>>(n, P, w.w, nullptr, w.s, Vj + n * P, w.active);
    }
    // u += Z_k s_k, s_k solving the rotated triangular system
    std::fill(hh.begin(), hh.end(), make_double2(0.0, 0.0));
    int kmax = 0;
    for (int p = 0; p < P; ++p) {
      if (!active[p] || kdim[p] == 0) continue;
      const int k = kdim[p];
      std::vector<cd> sv(k);
      for (int r = k - 1; r >= 0; --r) {
        cd acc = g[(size_t)p * (m + 1) + r];
        for (int c = r + 1; c < k; ++c) acc -= Hat(p, r, c) * sv[c];
        sv[r] = acc / Hat(p, r, r);
      }
      for (int r = 0; r < k; ++r) hh[(size_t)p * (kPitMaxRestart + 1) + r] = make_double2(sv[r].real(), sv[r].imag());
      if (k > kmax) kmax = k;
    }
    TP_CHECK_CUDA(cudaMemcpyAsync(w.active, active.data(), P * sizeof(int), cudaMemcpyHostToDevice, st));
    TP_CHECK_CUDA(cudaMemcpyAsync(w.h, hh.data(), hh.size() * sizeof(double2), cudaMemcpyHostToDevice, st));
    if (kmax > 0) {
      rc = S.combine(w.Z, kmax, 1.f, u);
      if (rc) return rc;
    }
  }
  // final true residuals
  std::fill(active.begin(), active.end(), 1);
  TP_CHECK_CUDA(cudaMemcpyAsync(w.active, active.data(), P * sizeof(int), cudaMemcpyHostToDevice, st));
  if (a->resid != nullptr) {
    rc = S.matvec(u, w.w);
    if (rc) return rc;
    pit_scale_kernel<<<pit_grid(n * P), kPitThreads, 0, st>>>(n, P, w.b, w.w, nullptr, w.w, w.active);
    rc = S.norms(w.w, rn);
    if (rc) return rc;
    for (int p = 0; p < P; ++p) a->resid[p] = std::sqrt(rn[p]);
  }
  if (a->iters != nullptr)
    for (int p = 0; p < P; ++p) a->iters[p] = iters[p];
  TP_CHECK_CUDA(cudaStreamSynchronize(st));
  return check_cuda(cudaGetLastError(), "tp_pit_solve");
}
