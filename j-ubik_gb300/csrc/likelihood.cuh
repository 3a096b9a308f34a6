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

// Whether two_quotients may form a / x: neither a quotient nor the residual a - x q leaves
// the normal range, so the residual is exact.  (b / x of a count b needs no more: b is 0
// or at least 1.)
__device__ __forceinline__ bool plain_quotient(float a, float x) {
  const float m = fabsf(x), n = fabsf(a);
  return m > 1e-18f && m < 1e18f && (n == 0.0f || (n > 1e-18f && n < 1e18f));
}

// a / x and b / x from one reciprocal, each quotient corrected by its residual (one
// Newton step on the quotient, Markstein 1990).  Tested for the bits of the division over
// that range of a and x; outside it, the division.
__device__ __forceinline__ void two_quotients(float a, float b, float x, float& qa, float& qb) {
  if (!plain_quotient(a, x)) {
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

// The same for two pairs of quotients.
__device__ __forceinline__ void two_quotients(float2 a, float2 b, float2 x, float2& qa,
                                              float2& qb) {
  if (!(plain_quotient(a.x, x.x) && plain_quotient(a.y, x.y))) {
    two_quotients(a.x, b.x, x.x, qa.x, qb.x);
    two_quotients(a.y, b.y, x.y, qa.y, qb.y);
    return;
  }
  float2 r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(x.x));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(x.y));
  const float2 m = make_float2(-x.x, -x.y);
  qa = pmul(a, r);
  qb = pmul(b, r);
  qa = pfma(pfma(m, qa, a), r, qa);
  qb = pfma(pfma(m, qb, b), r, qb);
}
__device__ __forceinline__ void two_quotients(double2 a, double2 b, double2 x, double2& qa,
                                              double2& qb) {
  two_quotients(a.x, b.x, x.x, qa.x, qb.x);
  two_quotients(a.y, b.y, x.y, qa.y, qb.y);
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

// Compensated sums of two sequences of values, or of products (fused with the
// compensation's subtraction): nc is minus Kahan's c.
template <typename T>
struct Kahan2 {
  cx<T> s = mkc<T>((T)0, (T)0), nc = mkc<T>((T)0, (T)0);
  __device__ __forceinline__ void add_y(cx<T> y) {
    const cx<T> t = padd(s, y);
    nc = psub(y, psub(t, s));
    s = t;
  }
  __device__ __forceinline__ void add(cx<T> v) { add_y(padd(v, nc)); }
  __device__ __forceinline__ void add_product(cx<T> a, cx<T> b) { add_y(pfma(a, b, nc)); }
  __device__ __forceinline__ double value() const {
    return ((double)s.x + (double)nc.x) + ((double)s.y + (double)nc.y);
  }
};

// Two pixels (of two image rows) at once, as poisson_px, from conv + low.
template <typename T>
__device__ __forceinline__ void poisson_px2(cx<T> conv, cx<T> low, cx<T> ep, const int32_t (&d)[2],
                                            cx<T>& w_o, cx<T>& res_o, Kahan2<T>& s_lam,
                                            Kahan2<T>& s_dlog) {
  const bool a = d[0] >= 0, b = d[1] >= 0;
  const cx<T> lam = pfma(ep, conv, pmul(ep, low));
  // pixels that are not read out: lam = 1 and a count of 0 enter nowhere
  const cx<T> x = mkc<T>(a ? lam.x : (T)1, b ? lam.y : (T)1);
  const cx<T> dd = mkc<T>(a ? (T)d[0] : (T)0, b ? (T)d[1] : (T)0);
  s_lam.add(mkc<T>(a ? lam.x : (T)0, b ? lam.y : (T)0));
  s_dlog.add_product(dd, mkc<T>(log(x.x), log(x.y)));
  cx<T> w, q;
  two_quotients(pmul(ep, ep), dd, x, w, q);
  const cx<T> res = pmul(ep, psub(both<T>((T)1), q));
  w_o = mkc<T>(a ? w.x : (T)0, b ? w.y : (T)0);
  res_o = mkc<T>(a ? res.x : (T)0, b ? res.y : (T)0);
}

}  // namespace jubik
