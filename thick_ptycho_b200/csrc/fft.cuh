// Shared-memory mixed-radix (8, 4, 2, 3, 5) Stockham FFT for one CTA.
//
// A transform of length n = 2^a 3^b 5^c lives in shared memory; each pass of
// radix R reads R values with stride n/R, applies the twiddles
// W_{Ns R}^{r k} (k = j mod Ns, Ns = product of the previous radices), does
// an R-point DFT in registers and writes them with stride Ns (autosort, so
// the result is in natural order without a bit-reversal pass).  Twiddles
// W_n^t = exp(-2 pi i t / n) are computed once per CTA in fp64 into shared
// memory.  Both directions are unnormalised (the inverse is n times
// numpy.fft.ifft); callers fold the 1/n into an adjacent multiply.
#pragma once

#include <type_traits>

#include "tp_common.cuh"

namespace tp {

constexpr int kFftMaxPasses = 12;
constexpr int kFftMaxN = 4096;

struct FftPlan {
  int n;
  int npass;
  int radix[kFftMaxPasses];
  // reciprocals of the passes' n / R and Ns (fast_div)
  uint32_t mt[kFftMaxPasses], ms[kFftMaxPasses];
};

// w / d for w d < 2^32 with m = fast_recip(d): the error of m, below one, adds
// less than w / 2^32 to the quotient, which is a multiple of 1 / d.
inline uint32_t fast_recip(uint32_t d) { return d == 1 ? 0u : (uint32_t)(((1ull << 32) + d - 1) / d); }
__device__ __forceinline__ int fast_div(int w, uint32_t m) { return m ? (int)__umulhi((uint32_t)w, m) : w; }

// Host: radices of n (8s first, then 4, 2, 3, 5); npass = 0 if unsupported.
inline FftPlan make_fft_plan(int n) {
  FftPlan p{};
  p.n = n;
  int m = n, k = 0;
  if (n < 1 || n > kFftMaxN) return p;
  while (m % 8 == 0 && k < kFftMaxPasses) { p.radix[k++] = 8; m /= 8; }
  while (m % 4 == 0 && k < kFftMaxPasses) { p.radix[k++] = 4; m /= 4; }
  while (m % 2 == 0 && k < kFftMaxPasses) { p.radix[k++] = 2; m /= 2; }
  while (m % 3 == 0 && k < kFftMaxPasses) { p.radix[k++] = 3; m /= 3; }
  while (m % 5 == 0 && k < kFftMaxPasses) { p.radix[k++] = 5; m /= 5; }
  p.npass = (m == 1) ? k : 0;
  int ns = 1;
  for (int i = 0; i < p.npass; ++i) {
    p.mt[i] = fast_recip((uint32_t)(n / p.radix[i]));
    p.ms[i] = fast_recip((uint32_t)ns);
    ns *= p.radix[i];
  }
  return p;
}

__device__ __forceinline__ void fft_twiddles(cx *tw, int n, int tid, int nth) {
  for (int t = tid; t < n; t += nth) {
    double s, c;
    sincospi(-2.0 * (double)t / (double)n, &s, &c);
    tw[t] = mkcx((rx)c, (rx)s);
  }
}

// a + b and a - b as one packed instruction each, the same roundings (additions of a
// term rotated by +-i stay scalar: the rotation is then a sign and a register name).
// The register transforms issue two thirds of the additions: a 3D multislice slice of
// 64 probes of 256 x 256 takes 42.4 us instead of 45.8, its adjoint 50.9 instead of 59.9.
#ifdef TP_C128_CHECK
__device__ __forceinline__ cx padd(cx a, cx b) { return cadd(a, b); }
__device__ __forceinline__ cx psub(cx a, cx b) { return csub(a, b); }
#else
__device__ __forceinline__ cx padd(cx a, cx b) {
  cx r;
  asm("{.reg .b64 p, q; mov.b64 p, {%2, %3}; mov.b64 q, {%4, %5}; add.rn.f32x2 p, p, q; mov.b64 {%0, %1}, p;}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ cx psub(cx a, cx b) {
  cx r;
  asm("{.reg .b64 p, q; mov.b64 p, {%2, %3}; mov.b64 q, {%4, %5}; sub.rn.f32x2 p, p, q; mov.b64 {%0, %1}, p;}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
#endif

// R-point DFT in place (sign = -1 forward, +1 inverse).
template <int R>
__device__ __forceinline__ void dft_small(cx (&v)[8], rx sign);

template <>
__device__ __forceinline__ void dft_small<2>(cx (&v)[8], rx) {
  const cx a = v[0], b = v[1];
  v[0] = padd(a, b);
  v[1] = psub(a, b);
}

// multiply by sign*i
__device__ __forceinline__ cx mul_si(cx z, rx sign) { return mkcx(-sign * z.y, sign * z.x); }

template <>
__device__ __forceinline__ void dft_small<4>(cx (&v)[8], rx sign) {
  const cx a0 = padd(v[0], v[2]), a1 = psub(v[0], v[2]);
  const cx b0 = padd(v[1], v[3]), b1 = mul_si(psub(v[1], v[3]), sign);
  v[0] = padd(a0, b0);
  v[2] = psub(a0, b0);
  v[1] = cadd(a1, b1);
  v[3] = csub(a1, b1);
}

template <>
__device__ __forceinline__ void dft_small<8>(cx (&v)[8], rx sign) {
  const rx h = TP_R(0.70710678118654752440);  // 1/sqrt(2)
  cx e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
  // 4-point DFTs of the even and odd samples
  cx a0 = padd(e[0], e[2]), a1 = psub(e[0], e[2]), b0 = padd(e[1], e[3]), b1 = mul_si(psub(e[1], e[3]), sign);
  e[0] = padd(a0, b0); e[2] = psub(a0, b0); e[1] = cadd(a1, b1); e[3] = csub(a1, b1);
  a0 = padd(o[0], o[2]); a1 = psub(o[0], o[2]); b0 = padd(o[1], o[3]); b1 = mul_si(psub(o[1], o[3]), sign);
  o[0] = padd(a0, b0); o[2] = psub(a0, b0); o[1] = cadd(a1, b1); o[3] = csub(a1, b1);
  // twiddles W8^k = exp(sign * i * pi k / 4)
  const cx w1 = mkcx(h, sign * h), w3 = mkcx(-h, sign * h);
  o[1] = cmul(o[1], w1);
  o[2] = mul_si(o[2], sign);
  o[3] = cmul(o[3], w3);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    v[k] = padd(e[k], o[k]);
    v[k + 4] = psub(e[k], o[k]);
  }
}

// 4-point DFT of (a0, a1, a2, a3) in place, X_m = sum_r a_r exp(sign 2 pi i r m / 4).
__device__ __forceinline__ void dft4_inplace(cx &a0, cx &a1, cx &a2, cx &a3, rx sign) {
  const cx s02 = padd(a0, a2), d02 = psub(a0, a2), s13 = padd(a1, a3);
  const cx jd13 = mul_si(psub(a1, a3), sign);
  a0 = padd(s02, s13);
  a2 = psub(s02, s13);
  a1 = cadd(d02, jd13);
  a3 = csub(d02, jd13);
}

// 16-point DFT as 4 x 4: with n = 4 n1 + n2 and m = k1 + 4 k2,
// X_m = sum_n2 W16^{n2 k1} W4^{n2 k2} sum_n1 x_{4 n1 + n2} W4^{n1 k1}:
// DFT-4 over n1 for every n2, twiddles W16^{n2 k1}, DFT-4 over n2 for every
// k1, then the 4 x 4 transpose of the output order.
__device__ __forceinline__ void dft16(cx (&v)[16], rx sign) {
  // cos and sin of 2 pi m / 16, m = 0..9 (the twiddle exponents n2 k1 used)
  constexpr rx kc[10] = {TP_R(1.0), TP_R(0.92387953251128675613), TP_R(0.70710678118654752440), TP_R(0.38268343236508977173), TP_R(0.0),
                            -TP_R(0.38268343236508977173), -TP_R(0.70710678118654752440), -TP_R(0.92387953251128675613), -TP_R(1.0),
                            -TP_R(0.92387953251128675613)};
  constexpr rx ks[10] = {TP_R(0.0), TP_R(0.38268343236508977173), TP_R(0.70710678118654752440), TP_R(0.92387953251128675613), TP_R(1.0),
                            TP_R(0.92387953251128675613), TP_R(0.70710678118654752440), TP_R(0.38268343236508977173), TP_R(0.0),
                            -TP_R(0.38268343236508977173)};
#pragma unroll
  for (int n2 = 0; n2 < 4; ++n2) dft4_inplace(v[n2], v[4 + n2], v[8 + n2], v[12 + n2], sign);
  // now v[4 k1 + n2] holds the inner DFT for (n2, k1)
#pragma unroll
  for (int k1 = 1; k1 < 4; ++k1)
#pragma unroll
    for (int n2 = 1; n2 < 4; ++n2) {
      const int m = n2 * k1;
      v[4 * k1 + n2] = cmul(v[4 * k1 + n2], mkcx(kc[m], sign * ks[m]));
    }
#pragma unroll
  for (int k1 = 0; k1 < 4; ++k1) dft4_inplace(v[4 * k1], v[4 * k1 + 1], v[4 * k1 + 2], v[4 * k1 + 3], sign);
  // v[4 k1 + k2] holds X_{k1 + 4 k2}: transpose
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = r + 1; c < 4; ++c) {
      const cx t = v[4 * r + c];
      v[4 * r + c] = v[4 * c + r];
      v[4 * c + r] = t;
    }
}

template <>
__device__ __forceinline__ void dft_small<3>(cx (&v)[8], rx sign) {
  const rx s3 = TP_R(0.86602540378443864676);  // sin(2 pi / 3)
  const cx t = cadd(v[1], v[2]);
  const cx d = mul_si(csub(v[1], v[2]), sign * s3);
  const cx m = mkcx(v[0].x - TP_R(0.5) * t.x, v[0].y - TP_R(0.5) * t.y);
  v[0] = cadd(v[0], t);
  v[1] = cadd(m, d);
  v[2] = csub(m, d);
}

template <>
__device__ __forceinline__ void dft_small<5>(cx (&v)[8], rx sign) {
  const rx c1 = TP_R(0.30901699437494742410), c2 = -TP_R(0.80901699437494742410);  // cos(2pi/5), cos(4pi/5)
  const rx s1 = TP_R(0.95105651629515357212), s2 = TP_R(0.58778525229247312917);   // sin(2pi/5), sin(4pi/5)
  const cx a1 = cadd(v[1], v[4]), b1 = csub(v[1], v[4]);
  const cx a2 = cadd(v[2], v[3]), b2 = csub(v[2], v[3]);
  const cx x0 = v[0];
  const cx m1 = mkcx(x0.x + c1 * a1.x + c2 * a2.x, x0.y + c1 * a1.y + c2 * a2.y);
  const cx m2 = mkcx(x0.x + c2 * a1.x + c1 * a2.x, x0.y + c2 * a1.y + c1 * a2.y);
  const cx n1 = mul_si(mkcx(s1 * b1.x + s2 * b2.x, s1 * b1.y + s2 * b2.y), sign);
  const cx n2 = mul_si(mkcx(s2 * b1.x - s1 * b2.x, s2 * b1.y - s1 * b2.y), sign);
  v[0] = cadd(x0, cadd(a1, a2));
  v[1] = cadd(m1, n1);
  v[4] = csub(m1, n1);
  v[2] = cadd(m2, n2);
  v[3] = csub(m2, n2);
}

// One pass; the twiddle exponent r k n / (Ns R) stays below n (k < Ns, r < R).
template <int R>
__device__ __forceinline__ void fft_pass(const cx *a, cx *b, int n, int Ns, uint32_t mt, uint32_t ms, const cx *tw,
                                         rx sign, int nb, int tid, int nth) {
  const int T = n / R;
  const int step = T / Ns;
  for (int w = tid; w < nb * T; w += nth) {
    const int bi = fast_div(w, mt), j = w - bi * T;
    const cx *src = a + bi * n;
    cx *dst = b + bi * n;
    const int jn = fast_div(j, ms), k = j - jn * Ns;
    cx v[8];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = src[j + r * T];
    if (Ns > 1) {
      const int ks = k * step;
#pragma unroll
      for (int r = 1; r < R; ++r) {
        const cx t = tw[r * ks];
        v[r] = cmul(v[r], mkcx(t.x, sign < 0 ? t.y : -t.y));
      }
    }
    dft_small<R>(v, sign);
    const int idx = jn * Ns * R + k;
#pragma unroll
    for (int r = 0; r < R; ++r) dst[idx + r * Ns] = v[r];
  }
}

// ------------------------------------------------------ fixed-size plans
// The passes with the length and the radix sequence known at compile time, so that
// every index division and modulo is by a constant: the Stockham form of the 3D
// preconditioner at the common transverse sizes, in a padded shared-memory layout.
// Element i of a
// transform sits at i + i/8 (one spare slot per 8 elements) and transform bi
// starts at bi * S, S = N + N/8 + 1.  The Stockham writes of the early passes
// (stride R elements) and column transposes (stride S) then spread over the
// shared-memory banks instead of hitting a few of them.
template <int N>
struct FftPad {
  static constexpr int S = N + N / 8 + 1;
};
__device__ __forceinline__ int fft_pad(int i) { return i + (i >> 3); }

template <int N, int Ns, int R>
__device__ __forceinline__ void fft_pass_padded(const cx *a, cx *b, const cx *tw, rx sign, int nb, int tid,
                                                int nth) {
  constexpr int T = N / R;
  constexpr int step = N / (Ns * R);
  constexpr int S = FftPad<N>::S;
  for (int w = tid; w < nb * T; w += nth) {
    const int bi = w / T, j = w - bi * T;
    const cx *src = a + bi * S;
    cx *dst = b + bi * S;
    const int k = j % Ns;
    cx v[R > 8 ? 16 : 8];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = src[fft_pad(j + r * T)];
#pragma unroll
    for (int r = 1; r < R; ++r) {
      const cx t = tw[(r * k * step) % N];
      v[r] = cmul(v[r], mkcx(t.x, sign < 0 ? t.y : -t.y));
    }
    if constexpr (R == 16) dft16(v, sign);
    else dft_small<R>(v, sign);
    const int idx = (j / Ns) * Ns * R + k;
#pragma unroll
    for (int r = 0; r < R; ++r) dst[fft_pad(idx + r * Ns)] = v[r];
  }
}

template <int N, int Ns, int R, int... Rest>
__device__ __forceinline__ cx *fft_run_padded(cx *a, cx *b, const cx *tw, rx sign, int nb, int tid,
                                                  int nth) {
  fft_pass_padded<N, Ns, R>(a, b, tw, sign, nb, tid, nth);
  __syncthreads();
  if constexpr (sizeof...(Rest) == 0) {
    return b;
  } else {
    return fft_run_padded<N, Ns * R, Rest...>(b, a, tw, sign, nb, tid, nth);
  }
}

// Radix 16 for 128 and 256, else 8s first, then 4, 2, 3.
// The fixed-size transforms in the padded layout (FftPad).
template <int N>
__device__ __forceinline__ cx *fft_block_padded(cx *a, cx *b, const cx *tw, bool inverse, int nb,
                                                    int tid, int nth) {
  const rx sign = inverse ? TP_R(1.0) : -TP_R(1.0);
  if constexpr (N == 32) return fft_run_padded<32, 1, 8, 4>(a, b, tw, sign, nb, tid, nth);
  else if constexpr (N == 64) return fft_run_padded<64, 1, 8, 8>(a, b, tw, sign, nb, tid, nth);
  else if constexpr (N == 128) return fft_run_padded<128, 1, 8, 16>(a, b, tw, sign, nb, tid, nth);
  else if constexpr (N == 192) return fft_run_padded<192, 1, 8, 8, 3>(a, b, tw, sign, nb, tid, nth);
  else if constexpr (N == 256) return fft_run_padded<256, 1, 16, 16>(a, b, tw, sign, nb, tid, nth);
  else return fft_run_padded<512, 1, 8, 8, 8>(a, b, tw, sign, nb, tid, nth);
}

// nb transforms of length pl.n stored back to back in `a` (scratch `b` of
// the same size).  Returns the buffer holding the result (a or b).  Ends
// with __syncthreads().
__device__ __forceinline__ cx *fft_block(cx *a, cx *b, const FftPlan &pl, const cx *tw, bool inverse,
                                             int nb, int tid, int nth) {
  const rx sign = inverse ? TP_R(1.0) : -TP_R(1.0);
  int Ns = 1;
  for (int ps = 0; ps < pl.npass; ++ps) {
    const int R = pl.radix[ps];
    switch (R) {
      case 8: fft_pass<8>(a, b, pl.n, Ns, pl.mt[ps], pl.ms[ps], tw, sign, nb, tid, nth); break;
      case 4: fft_pass<4>(a, b, pl.n, Ns, pl.mt[ps], pl.ms[ps], tw, sign, nb, tid, nth); break;
      case 2: fft_pass<2>(a, b, pl.n, Ns, pl.mt[ps], pl.ms[ps], tw, sign, nb, tid, nth); break;
      case 3: fft_pass<3>(a, b, pl.n, Ns, pl.mt[ps], pl.ms[ps], tw, sign, nb, tid, nth); break;
      default: fft_pass<5>(a, b, pl.n, Ns, pl.mt[ps], pl.ms[ps], tw, sign, nb, tid, nth); break;
    }
    __syncthreads();
    cx *t = a;
    a = b;
    b = t;
    Ns *= R;
  }
  return a;
}

// FFT of `rows` transforms of length n in shared memory: the compile-time
// plan in the padded layout when N > 0, else the runtime plan `pl`
// (unpadded).  Whole-CTA call.
template <int N>
__device__ __forceinline__ cx *fft_rows(cx *a, cx *b, const FftPlan &pl, const cx *tw, bool inverse,
                                            int rows) {
  if constexpr (N > 0) return fft_block_padded<N>(a, b, tw, inverse, rows, threadIdx.x, blockDim.x);
  else return fft_block(a, b, pl, tw, inverse, rows, threadIdx.x, blockDim.x);
}

// Shared-memory slot of element i of transform bi (length n).
template <int N>
__device__ __forceinline__ int fslot(int bi, int i, int n) {
  if constexpr (N > 0) return bi * FftPad<N>::S + fft_pad(i);
  else return bi * n + i;
}
// Shared-memory slots per transform.
template <int N>
__host__ __device__ constexpr int fstride(int n) {
  if constexpr (N > 0) return FftPad<N>::S;
  else return n;
}

__device__ __forceinline__ void load_twiddles(cx *tw, const cx *__restrict__ twg, int n) {
  for (int t = threadIdx.x; t < n; t += blockDim.x) tw[t] = twg[t];
}

// ------------------------------------------------ register four-step transforms
// A transform of length N = R1 * R2 with the short DFTs held in registers:
// with n = R2 n1 + n2 and k = k1 + R1 k2,
//   X[k1 + R1 k2] = sum_n2 W_R2^{n2 k2} W_N^{n2 k1} sum_n1 x[R2 n1 + n2] W_R1^{n1 k1}.
// Stage A (one thread per n2): the R1-point DFT over n1 in registers, the
// twiddles W_N^{n2 k1}, one write to shared memory; stage C (one thread per
// k1): one read, the R2-point DFT over n2, giving X[k1 + R1 k2].  An element
// passes through shared memory once (one write, one read) instead of once per
// Stockham pass plus the staging copies.  The inverse runs the stages in the
// opposite order with conjugate twiddles.  The twiddle table is padded like
// the transpose: W_N^{n2 k1} at k1 * (R2 + 1) + n2, so that both stages read
// it without bank conflicts.

// 12-point DFT as 4 x 3 (n = 3 n1 + n2, k = k1 + 4 k2), natural order in and out.
__device__ __forceinline__ void dft12(cx (&v)[16], rx sign) {
  const rx s3 = TP_R(0.86602540378443864676);  // sin(pi / 3)
  cx y[12];
#pragma unroll
  for (int n2 = 0; n2 < 3; ++n2) {
    cx a0 = v[n2], a1 = v[3 + n2], a2 = v[6 + n2], a3 = v[9 + n2];
    dft4_inplace(a0, a1, a2, a3, sign);
    y[4 * n2] = a0;
    y[4 * n2 + 1] = a1;
    y[4 * n2 + 2] = a2;
    y[4 * n2 + 3] = a3;
  }
  // W12^m = exp(sign 2 pi i m / 12) for m = n2 k1 in {1, 2, 3, 2, 4, 6}
  const cx w1 = mkcx(s3, sign * TP_R(0.5)), w2 = mkcx(TP_R(0.5), sign * s3), w3 = mkcx(TP_R(0.0), sign);
  const cx w4 = mkcx(-TP_R(0.5), sign * s3), w6 = mkcx(-TP_R(1.0), TP_R(0.0));
  y[5] = cmul(y[5], w1);
  y[6] = cmul(y[6], w2);
  y[7] = cmul(y[7], w3);
  y[9] = cmul(y[9], w2);
  y[10] = cmul(y[10], w4);
  y[11] = cmul(y[11], w6);
#pragma unroll
  for (int k1 = 0; k1 < 4; ++k1) {
    const cx a = y[k1], b = y[4 + k1], c = y[8 + k1];
    const cx t = padd(b, c);
    const cx d = mul_si(psub(b, c), sign * s3);
    const cx m = mkcx(a.x - TP_R(0.5) * t.x, a.y - TP_R(0.5) * t.y);
    v[k1] = padd(a, t);
    v[k1 + 4] = cadd(m, d);
    v[k1 + 8] = csub(m, d);
  }
}

// R-point DFT (R = 4, 8, 12, 16) of v[0..R) in registers, natural order in and out.
template <int R>
__device__ __forceinline__ void dft_reg(cx (&v)[16], rx sign) {
  static_assert(R == 4 || R == 8 || R == 12 || R == 16, "dft_reg: unsupported length");
  if constexpr (R == 16) {
    dft16(v, sign);
  } else if constexpr (R == 12) {
    dft12(v, sign);
  } else if constexpr (R == 8) {
    cx w[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) w[j] = v[j];
    dft_small<8>(w, sign);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = w[j];
  } else {
    dft4_inplace(v[0], v[1], v[2], v[3], sign);
  }
}

// ------------------------------------------------ in-place transforms, any 2^a 3^b 5^c
// For callers that multiply a spectrum and go back: the forward transform runs
// decimation-in-frequency stages in place (stage s splits blocks of len_s = n /
// (R_0 .. R_{s-1}) into R_s parts, str_s = len_s / R_s apart) and leaves the spectrum
// at p = k_0 str_0 + k_1 str_1 + ..., frequency k_0 + R_0 k_1 + R_0 R_1 k_2 + ...; the
// inverse undoes the stages in the opposite order.  A unit's R_s values keep their
// places, so a stage is one read and one write between two barriers and no pass
// reorders.
constexpr int kMixStages = 6;
struct MixPlan {
  int n, stages, threads, tw_total;
  int radix[kMixStages], len[kMixStages], str[kMixStages], tw[kMixStages];
  uint32_t ms[kMixStages];  // fast_div reciprocals of str
};

// The fewest stages with radices up to 16 and of those the most even split, the
// largest first, and at least two (n <= 16: a last one of radix 1); stages = 0 where
// there are none.
inline MixPlan make_mix_plan(int n) {
  MixPlan p{};
  p.n = n;
  if (n < 1 || n > kFftMaxN) return p;
  constexpr int radices[] = {16, 15, 12, 10, 9, 8, 6, 5, 4, 3, 2};
  int cur[kMixStages] = {}, best_len = kMixStages + 1, best_sum = 0;
  // non-increasing sequences of radices with product n (a few hundred nodes at most)
  auto search = [&](auto &self, int m, int k, int first, int sum) -> void {
    if (m == 1) {
      if (k < best_len || (k == best_len && sum < best_sum)) {
        best_len = k;
        best_sum = sum;
        for (int i = 0; i < k; ++i) p.radix[i] = cur[i];
      }
      return;
    }
    if (k >= kMixStages || k + 1 > best_len) return;
    for (int i = first; i < (int)(sizeof(radices) / sizeof(radices[0])); ++i)
      if (m % radices[i] == 0) {
        cur[k] = radices[i];
        self(self, m / radices[i], k + 1, i, sum + radices[i]);
      }
  };
  search(search, n, 0, 0, 0);
  if (n == 1) p.radix[best_len++] = 1;
  if (best_len > kMixStages) return p;
  if (best_len < 2) p.radix[best_len++] = 1;
  p.stages = best_len;
  int len = n, units = 0;
  for (int i = 0; i < p.stages; ++i) {
    p.len[i] = len;
    p.str[i] = len / p.radix[i];
    p.tw[i] = p.tw_total;
    p.ms[i] = fast_recip((uint32_t)p.str[i]);
    p.tw_total += i + 1 < p.stages ? len : 0;
    if (n / p.radix[i] > units) units = n / p.radix[i];
    len = p.str[i];
  }
  p.threads = (units + 31) / 32 * 32;
  return p;
}

// Slot of place i in shared memory: one spare per 16, so that the strides of the
// last stages (multiples of the radix) spread over the banks.
__host__ __device__ __forceinline__ int mix_pad(int i) { return i + (i >> 4); }
// Frequency at place p.
__device__ __forceinline__ int mix_frequency(const MixPlan &pl, int p) {
  int f = 0, mult = 1;
  for (int s = 0; s < pl.stages; ++s) {
    const int k = p / pl.str[s];
    p -= k * pl.str[s];
    f += mult * k;
    mult *= pl.radix[s];
  }
  return f;
}
// The stages' twiddles exp(-2 pi i k t / len_s) at tw[s] + k str_s + t (none for the last).
__device__ __forceinline__ void mix_twiddles(const MixPlan &pl, cx *tw, int tid, int nth) {
  for (int s = 0; s + 1 < pl.stages; ++s)
    for (int e = tid; e < pl.len[s]; e += nth) {
      const int k = e / pl.str[s], t = e - k * pl.str[s];
      double sv, cv;
      sincospi(-2.0 * (double)(k * t) / (double)pl.len[s], &sv, &cv);
      tw[pl.tw[s] + e] = mkcx((rx)cv, (rx)sv);
    }
}

// exp(2 pi i m / R), m < R, at compile time (Taylor series about 0 of an angle of at
// most pi / 4, quadrants by symmetry).
template <int R>
struct UnitRoots {
  rx c[R] = {}, s[R] = {};
  constexpr UnitRoots() {
    for (int m = 0; m < R; ++m) {
      int q = (8 * m + R) / (2 * R);  // nearest quarter turn
      const double x = 6.283185307179586476925 * ((double)(4 * m - q * R) / (4.0 * R));
      double cs = 1.0, sn = x, tc = 1.0, ts = x;
      for (int k = 1; k < 12; ++k) {
        tc *= -x * x / ((2 * k - 1) * (2 * k));
        ts *= -x * x / ((2 * k) * (2 * k + 1));
        cs += tc;
        sn += ts;
      }
      q &= 3;
      c[m] = (rx)(q == 0 ? cs : q == 1 ? -sn : q == 2 ? -cs : sn);
      s[m] = (rx)(q == 0 ? sn : q == 1 ? cs : q == 2 ? -sn : -cs);
    }
  }
};

// 3- and 5-point DFTs with their constants to twice the precision, c + (the rest of c):
// rounded, they are the same error in every slice of a march (255 slices of white noise
// at n = 1500: 2.1e-6 -> 1.9e-6; 64 probes 3.1 -> 3.3 us per slice).
template <int R>
__device__ __forceinline__ void dft_odd(cx (&v)[8], rx sign) {
#ifdef TP_C128_CHECK
  dft_small<R>(v, sign);
#else
  constexpr auto rest = [](double c) constexpr { return (float)(c - (double)(float)c); };
  if constexpr (R == 3) {
    constexpr double s = 0.86602540378443864676;  // sin(2 pi / 3)
    const cx t = padd(v[1], v[2]), b = psub(v[1], v[2]);
    const cx d = mul_si(mkcx(fmaf((float)s, b.x, rest(s) * b.x), fmaf((float)s, b.y, rest(s) * b.y)), sign);
    const cx m = mkcx(fmaf(-0.5f, t.x, v[0].x), fmaf(-0.5f, t.y, v[0].y));
    v[0] = padd(v[0], t);
    v[1] = cadd(m, d);
    v[2] = csub(m, d);
  } else {
    constexpr double c1 = 0.30901699437494742410, c2 = -0.80901699437494742410;  // cos(2 pi / 5), cos(4 pi / 5)
    constexpr double s1 = 0.95105651629515357212, s2 = 0.58778525229247312917;
    auto pair = [](double p, double q, float a, float b, float c) {  // c + p a + q b
      return fmaf((float)p, a, fmaf((float)q, b, fmaf(rest(p), a, fmaf(rest(q), b, c))));
    };
    const cx a1 = padd(v[1], v[4]), b1 = psub(v[1], v[4]);
    const cx a2 = padd(v[2], v[3]), b2 = psub(v[2], v[3]);
    const cx x0 = v[0];
    const cx m1 = mkcx(pair(c1, c2, a1.x, a2.x, x0.x), pair(c1, c2, a1.y, a2.y, x0.y));
    const cx m2 = mkcx(pair(c2, c1, a1.x, a2.x, x0.x), pair(c2, c1, a1.y, a2.y, x0.y));
    const cx n1 = mul_si(mkcx(pair(s1, s2, b1.x, b2.x, 0.f), pair(s1, s2, b1.y, b2.y, 0.f)), sign);
    const cx n2 = mul_si(mkcx(pair(s2, -s1, b1.x, b2.x, 0.f), pair(s2, -s1, b1.y, b2.y, 0.f)), sign);
    v[0] = padd(x0, padd(a1, a2));
    v[1] = cadd(m1, n1);
    v[4] = csub(m1, n1);
    v[2] = cadd(m2, n2);
    v[3] = csub(m2, n2);
  }
#endif
}
template <int R>
__device__ __forceinline__ void dft_part(cx (&v)[8], rx sign) {
  if constexpr (R == 3 || R == 5) dft_odd<R>(v, sign);
  else dft_small<R>(v, sign);
}

// R = A B points: n = B n1 + n2, k = k1 + A k2; A-point DFTs over n1, the roots
// exp(sign 2 pi i n2 k1 / R), B-point DFTs over n2.
template <int A, int B>
__device__ __forceinline__ void dft_two(cx (&v)[16], rx sign) {
  constexpr UnitRoots<A * B> w{};
  cx o[A * B];
#pragma unroll
  for (int n2 = 0; n2 < B; ++n2) {
    cx t[8];
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) t[n1] = v[B * n1 + n2];
    dft_part<A>(t, sign);
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1)
      o[B * k1 + n2] = n2 * k1 ? cmul(t[k1], mkcx(w.c[n2 * k1], sign * w.s[n2 * k1])) : t[k1];
  }
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) {
    cx t[8];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) t[n2] = o[B * k1 + n2];
    dft_part<B>(t, sign);
#pragma unroll
    for (int k2 = 0; k2 < B; ++k2) v[k1 + A * k2] = t[k2];
  }
}

// R-point DFT of v[0..R), R in {1, 2, 3, 4, 5, 6, 8, 9, 10, 12, 15, 16}.
template <int R>
__device__ __forceinline__ void mix_dft(cx (&v)[16], rx sign) {
  if constexpr (R == 16) dft16(v, sign);
  else if constexpr (R == 15) dft_two<3, 5>(v, sign);
  else if constexpr (R == 12) dft12(v, sign);
  else if constexpr (R == 10) dft_two<2, 5>(v, sign);
  else if constexpr (R == 9) dft_two<3, 3>(v, sign);
  else if constexpr (R == 6) dft_two<2, 3>(v, sign);
  else if constexpr (R > 1) {
    cx w[8];
#pragma unroll
    for (int j = 0; j < R; ++j) w[j] = v[j];
    dft_part<R>(w, sign);
#pragma unroll
    for (int j = 0; j < R; ++j) v[j] = w[j];
  }
}

// Calls f with the radix (at most RMAX) as a constant.
template <int RMAX, class F>
__device__ __forceinline__ void mix_radix(int radix, F f) {
  auto at = [&](auto r) {
    if constexpr (decltype(r)::value <= RMAX) f(r);
  };
  using std::integral_constant;
  switch (radix) {
    case 16: at(integral_constant<int, 16>{}); break;
    case 15: at(integral_constant<int, 15>{}); break;
    case 12: at(integral_constant<int, 12>{}); break;
    case 10: at(integral_constant<int, 10>{}); break;
    case 9: at(integral_constant<int, 9>{}); break;
    case 8: at(integral_constant<int, 8>{}); break;
    case 6: at(integral_constant<int, 6>{}); break;
    case 5: at(integral_constant<int, 5>{}); break;
    case 4: at(integral_constant<int, 4>{}); break;
    case 3: at(integral_constant<int, 3>{}); break;
    case 2: at(integral_constant<int, 2>{}); break;
    default: at(integral_constant<int, 1>{}); break;
  }
}

// Stage s of `count` elements (whole transforms, back to back, at mix_pad) in shared
// memory.  KIND 0: forward; 1: inverse; 2: the last stage, the product with h (by place)
// and its inverse; 3, 4: the last stage alone, forward and inverse (no twiddles).
template <int RMAX, int KIND>
__device__ __forceinline__ void mix_run(const MixPlan &pl, int s, int count, cx *buf, const cx *tw, const cx *h,
                                        int tid, int nth) {
  mix_radix<RMAX>(pl.radix[s], [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    constexpr bool LAST = KIND >= 2, INV = KIND == 1 || KIND == 4;
    const int str = LAST ? 1 : pl.str[s];
    for (int u = tid; u < count / R; u += nth) {
      int t = 0, base = u * R;
      if (!LAST) {
        const int b = fast_div(u, pl.ms[s]);
        t = u - b * str;
        base = b * (R * str) + t;
      }
      const cx *w = tw + pl.tw[s] + t;
      cx v[16];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        v[r] = buf[mix_pad(base + r * str)];
        if (KIND == 1 && r > 0) v[r] = cmulc(v[r], w[r * str]);
      }
      mix_dft<R>(v, INV ? TP_R(1.0) : -TP_R(1.0));
      if (KIND == 2) {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = cmul(v[r], h[base + r]);
        mix_dft<R>(v, TP_R(1.0));
      }
#pragma unroll
      for (int r = 0; r < R; ++r) buf[mix_pad(base + r * str)] = KIND == 0 && r > 0 ? cmul(v[r], w[r * str]) : v[r];
    }
  });
}

// ------------------------------------------- gain of a transform and its inverse
// A forward transform followed by the inverse that undoes its stages returns its input
// times n (1 + g): an element meets the same fp32 constants and twiddles in both
// directions, whose moduli are not quite one.  A march that multiplies a spectrum and
// goes back in every slice adds g (-8e-8 .. 9e-8) up; it folds 1 / (1 + g) into the
// spectrum's factor instead, which rounds once from fp64.  255 slices of white noise,
// error against complex128: n = 2048 3.7e-6 without it, 1.8e-6 with it; n = 1500 3.5e-6,
// 2.1e-6 (1.9e-6 with dft_odd's constants); 48 slices of 256 x 256: 1.8e-6, 8.8e-7.
//
// To first order g is a sum over the stages; this is the share of an R-point DFT's own
// constants (R of mix_dft and dft_reg).
template <int A, int B>
constexpr double root_gain() {
  const UnitRoots<A * B> w{};
  double g = 0.0;
  for (int a = 0; a < A; ++a)
    for (int b = 0; b < B; ++b) g += (double)w.c[a * b] * w.c[a * b] + (double)w.s[a * b] * w.s[a * b] - 1.0;
  return g / (A * B);
}
constexpr double dft_gain(int R) {
  constexpr double s3 = TP_R(0.86602540378443864676);  // rounded in dft12 only
  return R == 16 ? root_gain<4, 4>()
       : R == 15 ? root_gain<3, 5>()
       : R == 12 ? root_gain<4, 3>() + 4.0 * (s3 * s3 - 0.75) / 9.0
       : R == 10 ? root_gain<2, 5>()
       : R == 9  ? root_gain<3, 3>()
       : R == 8  ? root_gain<2, 4>()
       : R == 6  ? root_gain<2, 3>()
                 : 0.0;
}
inline double mix_dft_gain(const MixPlan &pl) {
  double g = 0.0;
  for (int s = 0; s < pl.stages; ++s) g += dft_gain(pl.radix[s]);
  return g;
}
__device__ __forceinline__ double modulus_less_1(cx w) { return (double)w.x * w.x + (double)w.y * w.y - 1.0; }
// This thread's part of the share of an in-place plan's twiddles (the table at tw).
__device__ __forceinline__ double mix_twiddle_gain(const MixPlan &pl, const cx *tw, int tid, int nth) {
  double g = 0.0;
  for (int s = 0; s + 1 < pl.stages; ++s) {
    double v = 0.0;
    for (int e = tid; e < pl.len[s]; e += nth) v += modulus_less_1(tw[pl.tw[s] + e]);
    g += v / pl.len[s];
  }
  return g;
}
// The sum of v over the CTA (whole warps, at most 32), for every thread; red: 32 values.
__device__ __forceinline__ double cta_sum(double v, double *red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
  __syncthreads();
  return s;
}

// Factors of the lengths with a four-step plan (R1 >= R2, both <= 16).
__host__ __device__ constexpr int four_r1(int n) { return n == 64 ? 8 : 16; }
__host__ __device__ constexpr int four_r2(int n) { return n / four_r1(n); }
__host__ __device__ constexpr bool four_step_size(int n) { return n == 64 || n == 128 || n == 192 || n == 256; }
// Entries of the padded twiddle table.
__host__ __device__ constexpr int four_tw_len(int n) { return four_r1(n) * (four_r2(n) + 1); }
// The gain's shares as above.
inline double four_dft_gain(int n) { return dft_gain(four_r1(n)) + dft_gain(four_r2(n)); }
__device__ __forceinline__ double four_twiddle_gain(int n, const cx *tw, int tid, int nth) {
  const int r2 = four_r2(n);
  double v = 0.0;
  for (int e = tid; e < n; e += nth) v += modulus_less_1(tw[e / r2 * (r2 + 1) + e % r2]);
  return v / n;
}

}  // namespace tp
