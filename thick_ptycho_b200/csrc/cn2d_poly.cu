// 2D Crank-Nicolson march of the 32-chunk layout with each slice solved by a fixed
// polynomial of its scaled off-diagonal part.
//
// In Cayley form a step needs e with (I - P_s) e = P_s v, v = u + src / 2 (exact
// adjoint: v = r + src): u_new = 2 (v + e) - u, and for the exact adjoint lambda = v +
// e, r_new = v + 2 e.  With D = I - diag(P_s) and J = D^{-1} offdiag(P_s), whose
// entries are i mu / D with mu ~ 0.02, e = p_m(J) D^{-1} P_s v for the Chebyshev
// residual polynomial of the segment [-i tau, i tau] (tau = the largest row sum of
// |J|, m = 6 at the paraxial sampling, cn3d_poly.cu has the same solve in 3D).  J
// couples only rows of opposite parity, so y_k of the Horner recurrence lives on the
// odd rows for even k and on the even rows for odd k, and the even half of e is one
// substitution.
//
// One CTA per probe.  A thread keeps R consecutive rows of the state for the whole
// march; a half-sweep's neighbours are its own rows and one warp shuffle.  Warps do
// not wait for one another inside a step: each computes H extra rows on both sides
// (what lies h rows outside changes a row by (tau / 2)^h, tau / 2 the largest entry of J;
// H = 8 rows leave 1e-13 at mu = 0.02 and 3e-10 at the largest mu taken, 0.056) and the halos are renewed through shared memory once per step, behind
// the step's only barrier.  The slices' diagonals (the QD rows of the factor set, in
// the layout of the stored field) are read one step ahead.  The partitioned
// solve it replaces runs one warp per probe through a chain of ceil(N / 32) dependent
// rows: N = 1201, 100 probes: 1.10 us per step against 3.40 (with the field kept 1.50
// against 4.18; exact adjoint with the gradient 2.4 against 31.4, whose sums went
// through shared-memory float atomics).
//
// The factorisation checks every row of a slice against the bounds the degree was
// chosen for and leaves the verdict in the slice; this kernel and the direct one
// (cn2d.cu) read those of the march's slices, and one of the two returns at once.
#include <math.h>

#include <complex>

#include "cn2d_internal.cuh"
#include "tp_errors.h"

#ifndef TP_C128_CHECK
namespace tp {

namespace {

constexpr int kHaloRows = 8;

struct Poly2DParams {
  MarchParams p;
  int M, nwarps, m;  // rows per chunk, warps per probe, degree
  float a[kPoly2DMaxDeg];
};

// i/(1 - qd), qd the diagonal of P.
__device__ __forceinline__ float2 ji_of(float2 qd) {
  const float dr = 1.f - qd.x, di = -qd.y;
  const float n = __fdividef(1.f, fmaf(dr, dr, di * di));
  return make_float2(di * n, dr * n);
}
// c + (J y)_i = c + Ji (wl y_{i-1} + wr y_{i+1})
__device__ __forceinline__ float2 jmul(float2 ji, float wl, float2 l, float wr, float2 r, float2 c) {
  const float sx = fmaf(wl, l.x, wr * r.x), sy = fmaf(wl, l.y, wr * r.y);
  return make_float2(fmaf(ji.x, sx, fmaf(-ji.y, sy, c.x)), fmaf(ji.x, sy, fmaf(ji.y, sx, c.y)));
}

// DEG: the degree when it is compiled in (its coefficients are then operands of the
// unrolled half-sweeps), else 0.
template <int R, int DEG, bool LAGGED, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) cn2d_poly_kernel(const __grid_constant__ Poly2DParams q) {
  static_assert(R % 2 == 0 && kHaloRows % R == 0, "whole lanes of halo");
  constexpr int HL = kHaloRows / R, USE = (32 - 2 * HL) * R;  // halo lanes, rows a warp owns
  constexpr int EX = HL * R;
  const MarchParams &p = q.p;
  extern __shared__ __align__(16) float2 ex[];  // [2][nwarps][2][EX]
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int g0 = w * USE + (lane - HL) * R;  // first row of this lane
  const bool own = lane >= HL && lane < 32 - HL;
  const size_t probe = blockIdx.x;
  const bool do_grad = LAGGED && p.grad_c != nullptr;

  int off[R];  // place of row g0 + i in a chunked slice (clamped outside)
  float wl[R], wr[R];
  unsigned in = 0, put = 0;  // rows of the matrix; rows this lane stores (with the padding)
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int g = g0 + i;
    const bool row = g >= 0 && g < p.N;
    const int gc = min(max(g, 0), p.Npad - 1);
    off[i] = (gc % q.M) * 32 + gc / q.M;
    if (row) in |= 1u << i;
    if (own && g < p.Npad) put |= 1u << i;
    wl[i] = !row || g == 0 ? 0.f : (g == p.N - 1 ? p.sp.subN1.y : (g == 1 ? p.sp.sub1.y : p.sp.p_o.y));
    wr[i] = !row || g == p.N - 1 ? 0.f : (g == 0 ? p.sp.sup0.y : (g == p.N - 2 ? p.sp.supN2.y : p.sp.p_o.y));
  }
  if (lane == 0) wl[0] = 0.f;  // beyond the halo
  if (lane == 31) wr[R - 1] = 0.f;
  pdl_trigger();
  pdl_wait();

  auto slice_of = [&](int t) { return p.backward ? (p.L + 1 - t) : t; };
  auto diag = [&](int t, float2(&d)[R]) {
    const float2 *src = reinterpret_cast<const float2 *>(p.factors + (size_t)(slice_of(t) - 1) * p.slice_bytes);
#pragma unroll
    for (int i = 0; i < R; ++i) d[i] = src[off[i]];
  };
  const float2 zero = make_float2(0.f, 0.f);
  float2 u[R], qd[R], qn[R], f1[R], f0[R];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    u[i] = f1[i] = f0[i] = zero;
    if (!((in >> i) & 1u)) continue;
    if (p.state_in != nullptr) u[i] = p.state_in[probe * p.state_stride + off[i]];
    else if (p.probes != nullptr && p.t0 == 1) u[i] = p.probes[probe * p.N + g0 + i];
  }
  diag(p.t0, qn);  // (on their way while the verdicts are read)
  // The halo rows belong to neighbouring warps, whose outputs may replace the inputs
  // (state_out or exit_out on state_in, probes or a source): every warp has read before
  // one writes, by the barrier in here.  A march of several steps has the halos' barriers
  // in between.
  if (poly_excluded(p)) return;  // the direct kernel runs this march
  auto store = [&](float2 *dst, const float2(&v)[R]) {
#pragma unroll
    for (int i = 0; i < R; ++i)
      if ((put >> i) & 1u) dst[off[i]] = v[i];
  };
  if (p.u_store != nullptr && store_index(p, p.t0 - 1) >= 0)
    store(p.u_store + (probe * p.store_slices + store_index(p, p.t0 - 1)) * p.Npad, u);
  auto forward_slice = [&](int s, float2(&f)[R]) {
    const float2 *src = p.u_fwd + (probe * p.ufwd_slices + (s - p.ufwd_base)) * p.Npad;
#pragma unroll
    for (int i = 0; i < R; ++i)
      if (own && ((in >> i) & 1u)) f[i] = src[off[i]];
  };
  if (do_grad) forward_slice(slice_of(p.t0), f1);
  const bool sources = p.src_shared != nullptr || p.src_probe != nullptr || p.src_exit != nullptr;
  auto add_sources = [&](int t, float sw, float2(&v)[R]) {
    const float2 *s0 = p.src_shared ? p.src_shared + (size_t)(t - 1) * p.N + g0 : nullptr;
    const float2 *s1 =
        p.src_probe ? p.src_probe + (probe * p.L + (p.src_rev ? p.L - t : t - 1)) * p.N + g0 : nullptr;
    const float2 *s2 = (t == 1 && p.src_exit) ? p.src_exit + probe * p.N + g0 : nullptr;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      if (!((in >> i) & 1u)) continue;
      if (s0) v[i] = caxpy(sw, s0[i], v[i]);
      if (s1) v[i] = caxpy(sw, s1[i], v[i]);
      if (s2) v[i] = caxpy(sw, s2[i], v[i]);
    }
  };

  for (int t = p.t0; t <= p.t1; ++t) {
    const int s = slice_of(t);
#pragma unroll
    for (int i = 0; i < R; ++i) qd[i] = ((in >> i) & 1u) ? qn[i] : zero;
    if (t < p.t1) diag(t + 1, qn);
    if (do_grad) forward_slice(s - 1, f0);
    if (sources) add_sources(t, LAGGED ? 1.f : 0.5f, u);
    // g = D^{-1} P v; D^{-1} b = b + qd (D^{-1} b) keeps the operator's 1 + eps form
    float2 ji[R], g[R];
    {
      const float2 left = shfl_up2(u[R - 1], 1), right = shfl_down2(u[0], 1);
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const float2 l = i > 0 ? u[i > 0 ? i - 1 : 0] : left, r = i + 1 < R ? u[i + 1 < R ? i + 1 : i] : right;
        const float sx = fmaf(wl[i], l.x, wr[i] * r.x), sy = fmaf(wl[i], l.y, wr[i] * r.y);
        const float2 b = make_float2(fmaf(qd[i].x, u[i].x, fmaf(-qd[i].y, u[i].y, -sy)),
                                     fmaf(qd[i].x, u[i].y, fmaf(qd[i].y, u[i].x, sx)));
        ji[i] = ji_of(qd[i]);
        const float2 d = make_float2(fmaf(ji[i].y, b.x, ji[i].x * b.y), fmaf(ji[i].y, b.y, -ji[i].x * b.x));
        g[i] = cfma(qd[i], d, b);
      }
    }
    // y_k on even rows (odd k) and odd rows (even k) in e[]
    float2 e[R];
    {
      const float am = q.a[(DEG > 0 ? DEG : q.m) - 1];
#pragma unroll
      for (int i = 0; i < R; i += 2) e[i] = make_float2(am * g[i].x, am * g[i].y);
    }
    auto pair = [&](int k) {
      {
        const float a = q.a[k];
        const float2 right = shfl_down2(e[0], 1);
#pragma unroll
        for (int i = 1; i < R; i += 2) {
          const float2 r = i + 1 < R ? e[i + 1 < R ? i + 1 : 0] : right;
          e[i] = jmul(ji[i], wl[i], e[i - 1], wr[i], r, make_float2(a * g[i].x, a * g[i].y));
        }
      }
      {
        const float a = k > 0 ? q.a[k - 1] : 1.f;
        const float2 left = shfl_up2(e[R - 1], 1);
#pragma unroll
        for (int i = 0; i < R; i += 2) {
          const float2 l = i > 0 ? e[i > 0 ? i - 1 : 0] : left;
          e[i] = jmul(ji[i], wl[i], l, wr[i], e[i + 1], make_float2(a * g[i].x, a * g[i].y));
        }
      }
    };
    if constexpr (DEG > 0) {
#pragma unroll
      for (int k = DEG - 2; k >= 0; k -= 2) pair(k);
    } else {
#pragma unroll 1
      for (int k = q.m - 2; k >= 0; k -= 2) pair(k);
    }
    // the last step's outputs, the same for its sources
    auto sources_read = [&]() {
      if (sources && t == p.t1) __syncthreads();
    };
    float2 *dst = nullptr;
    if (p.u_store != nullptr && store_index(p, t) >= 0)
      dst = p.u_store + (probe * p.store_slices + store_index(p, t)) * p.Npad;
    if constexpr (LAGGED) {
      float2 lam[R];
#pragma unroll
      for (int i = 0; i < R; ++i) lam[i] = cadd(u[i], e[i]);
      sources_read();
      if (dst) store(dst, lam);
      if (t == p.L && p.exit_out != nullptr) {
#pragma unroll
        for (int i = 0; i < R; ++i)
          if (own && ((in >> i) & 1u)) p.exit_out[probe * p.N + g0 + i] = lam[i];
      }
      if (do_grad) {
        float2 *gr = p.grad_c + (size_t)(s - 1) * p.Npad;
#pragma unroll
        for (int i = 0; i < R; ++i) {
          if (own && ((in >> i) & 1u)) red_add_cx(&gr[off[i]], cmulc(lam[i], cadd(f1[i], f0[i])));
          f1[i] = f0[i];
        }
      }
    }
#pragma unroll
    for (int i = 0; i < R; ++i) u[i] = caxpy(2.f, e[i], u[i]);
    if constexpr (!LAGGED) {
      if (sources) add_sources(t, 0.5f, u);
      sources_read();
      if (dst) store(dst, u);
      if (t == p.L && p.exit_out != nullptr) {
#pragma unroll
        for (int i = 0; i < R; ++i)
          if (own && ((in >> i) & 1u)) p.exit_out[probe * p.N + g0 + i] = u[i];
      }
    }
    if (t == p.t1) break;
    // renew the halos from the neighbouring warps' rows
    if (q.nwarps > 1) {
      float2 *mine = ex + (((t & 1) * q.nwarps + w) * 2) * EX;
      if (lane >= HL && lane < 2 * HL) {
#pragma unroll
        for (int i = 0; i < R; ++i) mine[(lane - HL) * R + i] = u[i];
      }
      if (lane >= 32 - 2 * HL && lane < 32 - HL) {
#pragma unroll
        for (int i = 0; i < R; ++i) mine[EX + (lane - (32 - 2 * HL)) * R + i] = u[i];
      }
      __syncthreads();
      if (lane < HL && w > 0) {
        const float2 *src = mine - 2 * EX + EX + lane * R;  // warp w - 1's last rows
#pragma unroll
        for (int i = 0; i < R; ++i) u[i] = src[i];
      }
      if (lane >= 32 - HL && w + 1 < q.nwarps) {
        const float2 *src = mine + 2 * EX + (lane - (32 - HL)) * R;  // warp w + 1's first rows
#pragma unroll
        for (int i = 0; i < R; ++i) u[i] = src[i];
      }
    }
  }
  if (p.state_out != nullptr) store(p.state_out + probe * p.Npad, u);
}

template <int R, bool LAGGED, int MAXT, int MINB>
int launch(const Poly2DParams &q, cudaStream_t st) {
  constexpr int HL = kHaloRows / R;
  const size_t smem = (size_t)4 * q.nwarps * HL * R * sizeof(float2);
  auto kern = q.m == 6 ? cn2d_poly_kernel<R, 6, LAGGED, MAXT, MINB> : cn2d_poly_kernel<R, 0, LAGGED, MAXT, MINB>;
  return check_cuda(launch_dependent(kern, dim3(q.p.P), dim3(32 * q.nwarps), smem, st, true, q), "cn2d_poly_kernel launch");
}

std::complex<double> chebyshev(int m, std::complex<double> w) {
  std::complex<double> t0 = 1.0, t1 = w;
  for (int j = 1; j < m; ++j) {
    const std::complex<double> t2 = 2.0 * w * t1 - t0;
    t0 = t1;
    t1 = t2;
  }
  return t1;
}

}  // namespace

Poly2DPlan poly2d_plan(const tp_cn2d_op *op) {
  Poly2DPlan pl{};
  if (op->k_off[0] != 0.0 || op->k_01[0] != 0.0 || op->k_nm[0] != 0.0) return pl;
  const double mu = fabs(op->k_off[1]);
  const double dr = 1.0 - op->k_diag[0], di = op->k_diag[1], d = hypot(dr, di);
  if (!(d > 0.5)) return pl;
  // margins over the free-space slice for the object and the boundary rows
  const double tau = 1.15 * 2.0 * mu / d + 0.002;
  // halo rows leave 3e-10 of what lies beyond them (rows within tau couple by at most
  // tau / 2 to either side, but for the doubled couplings of the edges)
  if (!(pow(0.5 * tau, (double)kHaloRows) <= 3.3e-10)) return pl;
  double arg = fabs(atan2(di, dr)) + 0.1;
  if (!(arg < 1.5)) return pl;  // the factorisation compares tangents
  const std::complex<double> it(0.0, tau);
  for (int m = 4; m <= kPoly2DMaxDeg; m += 2) {
    const std::complex<double> scale = chebyshev(m, 1.0 / it);
    auto holds = [&](double x) { return std::abs(chebyshev(m, std::polar(1.0, x))) <= 3e-8 * std::abs(scale); };
    if (!holds(arg)) continue;
    // the widest object the degree covers: |n - 1| up to 0.08 at wavelength 0.5 with unit
    // steps (m = 6), against 0.016 at the first margin
    while (arg < 1.2 && holds(arg + 0.05)) arg += 0.05;
    double t0[kPoly2DMaxDeg + 1] = {1.0}, t1[kPoly2DMaxDeg + 1] = {0.0, 1.0};
    for (int n = 1; n < m; ++n) {
      double t2[kPoly2DMaxDeg + 1] = {0.0};
      for (int j = 0; j <= m; ++j) t2[j] = (j > 0 ? 2.0 * t1[j - 1] : 0.0) - t0[j];
      for (int j = 0; j <= m; ++j) t0[j] = t1[j], t1[j] = t2[j];
    }
    std::complex<double> pw = 1.0, sum = 1.0;  // (i tau)^{-j}
    for (int k = 0; k < m; ++k) {
      sum -= t1[k] * pw / scale;
      pl.a[k] = (float)sum.real();
      pw /= it;
    }
    pl.m = m;
    pl.tau_max = (float)tau;
    pl.arg_max = (float)arg;
    return pl;
  }
  return pl;
}

int launch_poly_march(const Partition &pt, const MarchParams &mp, const Poly2DPlan &plan, bool lagged, cudaStream_t st) {
  Poly2DParams q{};
  q.p = mp;
  q.M = pt.M;
  q.m = plan.m;
  for (int k = 0; k < plan.m; ++k) q.a[k] = plan.a[k];
  auto warps = [&](int R) {
    const int use = 32 * R - 2 * kHaloRows;
    return (mp.Npad + use - 1) / use;
  };
  // Fewer rows per thread shorten a step's dependent chain but add halo rows and warps:
  // 2 (then 4) while the matrix takes at most ten warps, else 8 (us per step to the exit
  // with 2, 4, 8 rows: N = 256, 32 probes 0.69, 0.75, 0.78; 777, 64: 1.44, 1.08, 1.09;
  // 1201, 100: -, 1.40, 1.10).  With more probes than SMs, up to seven warps, two CTAs per
  // SM at 128 registers (1500, 300 probes: 3.25 -> 2.96; the exact adjoint would spill).
  if (warps(2) <= 10) {
    q.nwarps = warps(2);
    return lagged ? launch<2, true, 320, 3>(q, st) : launch<2, false, 320, 3>(q, st);
  }
  if (warps(4) <= 10) {
    q.nwarps = warps(4);
    return lagged ? launch<4, true, 320, 2>(q, st) : launch<4, false, 320, 2>(q, st);
  }
  q.nwarps = warps(8);
  int dev = 0, sms = 148;
  TP_CHECK_CUDA(cudaGetDevice(&dev));
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (q.nwarps <= 7 && !lagged && mp.P > sms) return launch<8, false, 224, 2>(q, st);
  return lagged ? launch<8, true, 288, 1>(q, st) : launch<8, false, 288, 1>(q, st);
}

}  // namespace tp
#endif  // TP_C128_CHECK
