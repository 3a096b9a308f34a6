// Per-pixel Poisson terms and their deterministic reductions, shared by the
// image-space likelihood pass (ops.cu) and the row kernels (sep_rows.cuh).
#pragma once

#include <cstdint>

#include "jubik_common.cuh"

namespace jubik {

// Compensated (Kahan) accumulation in the working precision.
template <typename T>
struct Kahan {
  T s = (T)0, c = (T)0;
  __device__ __forceinline__ void add(T v) {
    const T y = v - c;
    const T t = s + y;
    c = (t - s) - y;
    s = t;
  }
  __device__ __forceinline__ double value() const { return (double)s - (double)c; }
};

// Block sums of (a, b) into partials[bid] (sa, sb: shared scratch of blockDim.x
// doubles each); the last of nblocks blocks to finish sums the partials in a
// fixed order (deterministic) and writes a - b.
__device__ __forceinline__ void block_reduce2_of(double a, double b, double* sa, double* sb,
                                                 double* partials, unsigned int* counter,
                                                 double* energy, unsigned int bid,
                                                 unsigned int nblocks) {
  __shared__ bool last;
  // pairwise tree over the largest power of two below the block size
  int top = 1;
  while (2 * top < (int)blockDim.x) top *= 2;
  auto tree = [&](double x, double y) {
    sa[threadIdx.x] = x;
    sb[threadIdx.x] = y;
    __syncthreads();
    for (int w = top; w > 0; w >>= 1) {
      if ((int)threadIdx.x < w && threadIdx.x + w < blockDim.x) {
        sa[threadIdx.x] += sa[threadIdx.x + w];
        sb[threadIdx.x] += sb[threadIdx.x + w];
      }
      __syncthreads();
    }
  };
  tree(a, b);
  if (threadIdx.x == 0) {
    partials[2 * bid] = sa[0];
    partials[2 * bid + 1] = sb[0];
    __threadfence();
    const unsigned int done = atomicAdd(counter, 1u);
    last = (done == nblocks - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double p1 = 0.0, p2 = 0.0;
  for (unsigned int i = threadIdx.x; i < nblocks; i += blockDim.x) {
    p1 += __ldcg(partials + 2 * i);
    p2 += __ldcg(partials + 2 * i + 1);
  }
  tree(p1, p2);
  if (threadIdx.x == 0) {
    // H = sum(lam) - vdot(d, log(lam))
    if (energy) energy[0] = sa[0] - sb[0];
    *counter = 0u;
  }
}

// a / x and b / x from one reciprocal, each quotient corrected by its residual (one
// Newton step on the quotient, Markstein 1990): within rounding of the exact
// quotients for x of ordinary size; others divide.
__device__ __forceinline__ void two_quotients(float a, float b, float x, float& qa, float& qb) {
  const bool plain = fabsf(x) > 1e-18f && fabsf(x) < 1e18f && fabsf(a) < 1e18f;
  if (!plain) {
    qa = a / x;
    qb = b / x;
    return;
  }
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  qa = a * r;
  qb = b * r;
  qa = fmaf(fmaf(-x, qa, a), r, qa);
  qb = fmaf(fmaf(-x, qb, b), r, qb);
}
__device__ __forceinline__ void two_quotients(double a, double b, double x, double& qa,
                                              double& qb) {
  qa = a / x;
  qb = b / x;
}

// One pixel: lam = eps * conv where a pixel is read out (count >= 0), the
// energy terms, the residual eps * (1 - d/lam) (0 elsewhere) and the metric
// weight eps^2 / lam (0 elsewhere) that later Fisher-metric products apply to
// R v: the image-space weights of R^T diag(1/lam) R (the exposure enters once
// from R and once from R^T).
template <typename T>
__device__ __forceinline__ void poisson_px(T conv, T ep, int32_t d, T& w_o, T& res_o,
                                           Kahan<T>& s_lam, Kahan<T>& s_dlog) {
  if (d < 0) {
    res_o = (T)0;
    w_o = (T)0;
    return;
  }
  const T lam = ep * conv;
  const T dd = (T)d;
  s_lam.add(lam);
  s_dlog.add(dd * log(lam));
  T q;
  two_quotients(ep * ep, dd, lam, w_o, q);
  res_o = ep * ((T)1 - q);
}

}  // namespace jubik
