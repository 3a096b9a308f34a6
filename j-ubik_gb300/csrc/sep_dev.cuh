// Device helpers shared by the separable row and column kernels.
#pragma once

#include <algorithm>
#include <mutex>
#include <vector>

#include "fft_codelets.cuh"
#include "sep.h"

namespace jubik {
namespace {

// Programmatic dependent launch: let the next kernel be scheduled, and wait for
// the previous kernel before touching anything it writes.  Loads of what an
// earlier kernel of the chain wrote are plain loads: read-only loads (__ldg,
// __restrict__) may be moved above the wait.
__device__ __forceinline__ void sep_trigger() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void sep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// floor(u / d) for u >= 0 by one multiply-high (mul from mulhi_divisor; 0: divide)
__device__ __forceinline__ int sep_div(int u, int d, uint32_t mul) {
  return mul ? (int)__umulhi((uint32_t)u, mul) : u / d;
}

// a + conj(b) and (a - conj(b)) / i: twice the spectra of the two real rows of a
// pair from the pair's transform at k and -k (the rows are halved before)
template <typename T>
__device__ __forceinline__ cx<T> split_a(cx<T> a, cx<T> b) {
  return mkc<T>(a.x + b.x, a.y - b.y);
}
template <typename T>
__device__ __forceinline__ cx<T> split_b(cx<T> a, cx<T> b) {
  return mkc<T>(a.y + b.y, b.x - a.x);
}

// twiddles q and q + 1 (q even) of a class in one 16-byte load (FP32)
__device__ __forceinline__ void two_twiddles(const float2* tw, int q, float2& a, float2& b) {
  const float4 t = *reinterpret_cast<const float4*>(tw + q);
  a = make_float2(t.x, t.y);
  b = make_float2(t.z, t.w);
}
__device__ __forceinline__ void two_twiddles(const double2* tw, int q, double2& a, double2& b) {
  a = tw[q];
  b = tw[q + 1];
}

// s + e = a + b exactly, part by part (Knuth's TwoSum)
template <typename C>
__device__ __forceinline__ void two_sum(C a, C b, C& s, C& e) {
  s = padd(a, b);
  const C t = psub(s, a);
  e = padd(psub(a, psub(s, t)), psub(b, t));
}

// Per kernel: the shared-memory opt-in raised so far and the CTAs that fit an
// SM, per device and size (looked up once, so never inside a stream capture
// that follows a first call of the same shapes).
struct SepKernelCache {
  struct Entry {
    int dev, threads;
    size_t smem;
    int per_sm;
  };
  std::mutex mu;
  std::vector<Entry> seen;
  int prepare(const void* kern, int threads, size_t smem, int* per_sm) {
    int dev = 0;
    JUBIK_TRY_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    size_t top = 0;
    for (const Entry& e : seen) {
      if (e.dev != dev) continue;
      if (e.smem == smem && e.threads == threads) {
        *per_sm = e.per_sm;
        return JUBIK_OK;
      }
      top = std::max(top, e.smem);
    }
    if (smem > top)  // the attribute only ever grows: another size may be in use
      JUBIK_TRY_CUDA(
          cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int n = 0;
    JUBIK_TRY_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, threads, smem));
    *per_sm = std::max(1, n);
    seen.push_back(Entry{dev, threads, smem, *per_sm});
    return JUBIK_OK;
  }
};

template <typename KernelT, typename... ArgsT>
int sep_launch(KernelT kern, dim3 grid, int threads, size_t smem, bool pdl, cudaStream_t s,
               const char* what, ArgsT... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cuda_status(cudaLaunchKernelEx(&cfg, kern, args...), what);
}

}  // namespace
}  // namespace jubik
