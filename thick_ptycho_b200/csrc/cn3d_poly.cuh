// The polynomial form of the 3D Crank-Nicolson march (cn3d_poly.cu).
#pragma once

#include <cuda_runtime.h>

#include "tp_common.cuh"

namespace tp {

// One march, in the terms of tp_cn3d_march: the diagonals are those of
// sigma*T(K), vec[0] holds the initial state and vec[1] is the vector `vstride`
// bytes after it (the states alternate between the two), scratch and the
// small arrays are workspace that nothing else uses during the march.
struct C3PolyJob {
  int nf, nb, nz, P;
  int mode, exact, is_delta, dtype, conj_t;
  double sigma, k, dz, tol;
  int max_iter;
  double mu_x, mu_y;  // imaginary interior couplings of sigma*T(K)
  const void *field;
  const float2 *kc, *kw, *ke, *ks, *kn;
  float2 *vec[2];
  size_t vstride;
  char *scratch;
  size_t scratch_bytes;
  float2 *colw;  // (nf)
  float4 *roww;  // (nb)
  int *check;    // 5 words
  const float2 *probes, *src_exit, *src_shared, *u_fwd;
  float2 *u_store, *exit_out, *grad_c;
  int *stats;
  int sums;  // u_store and u_fwd hold pair sums u_s + u_{s-1} at s
};

// Widths up to this many rows or columns fit the small arrays.
constexpr int kPolyMaxSide = 2048;

// The smallest even degree m <= max_m whose residual polynomial stays below `target`
// on the segment [-i tau, i tau] turned by up to `theta` (0: none); a[k], k < m, are the
// coefficients of p_m.
int poly_degree(double tau, double theta, double target, int max_m, float *a);

// Runs the march if its operator allows the polynomial form (*ran = 1);
// otherwise leaves it to the Krylov march (*ran = 0, nothing written that the
// Krylov march reads).  Waits once for `stream`, before the first step.
int c3_poly_march(const C3PolyJob &job, cudaStream_t stream, int *ran);

}  // namespace tp
