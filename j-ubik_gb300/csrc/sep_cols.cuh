// Column kernels of the separable response (see sep.h).
//
// A CTA holds CG adjacent columns (kx) of one patch, P rows each, in shared
// memory.  A column transform of side P = 16 L1 is a two-phase four-step:
//   forward: DFT-L1 over rows n2 + 16 i, then DFT-16 per class with twiddles;
//            the spectrum of class cls sits in registers, X[cls + L1 q], the
//            order of the stored PSF spectra (slot 16 cls + q);
//   inverse: DFT-16 per class, twiddles, then DFT-L1: rows 16 i + q in natural
//            order.
// Column 0 carries the packed kx = 0 and kx = P/2 columns: its product with the
// PSF is alpha W(ky) + beta conj(W(-ky)) (conjugated coefficients for the
// adjoint), with W(-ky) exchanged through shared memory.
//
// CG = 8 columns give row segments of 64 bytes (FP32) and CTAs of a few warps, so
// that 16 warps share an SM in independent CTAs: one CTA's loads overlap another's
// transforms.  Within a CTA the PSF spectra (and the adjoint's rows) are loaded
// into registers one transform ahead.  The kernels are bound by the LSU data
// pipe (forward 47 %, adjoint 56 % busy at 512^2: the exchange between the two phases, the
// twiddles, the loads) together with instruction issue (43 and 48 %), beside DRAM: at
// 1024^2 x 7 x 3 the forward moves 1297 MB in 288 us (4.5 TB/s), the adjoint
// 1194 MB in 243 us (4.9 TB/s of a copy's 6.8); the per-patch kernels before
// them took 519 and 511 us.  The module sum stays in registers (250 us; 306 in
// tensor memory); the rows that later patches of a run also cover wait in tensor
// memory (TMEM, 128 lanes x 512 columns per SM, otherwise unused), which costs
// neither registers nor LSU cycles.
//
// The next kernel is let in at the end of a CTA's work, not at its start: row CTAs
// that enter beside running column CTAs find the shared memory fragmented, so that
// some SMs took two of them and others five (three fit), and the last of the looping
// CTAs started when the first ended: 1173 us for a pass at 1024^2 x 7 x 3 against 923.
#include "sep_dev.cuh"

namespace jubik {
namespace {

struct ColK {
  SepCols a;
  int M, E, nx, n, n2, dx, half, margin, sr_max, K;
  int nq;        // runs per patch column
  int mc;        // modules per CTA (runs of patches)
  uint32_t div_n2, div_n, div_q;
};

constexpr int kColGroup = 8;

template <typename T, int L1>
struct ColT {
  static constexpr int P = 16 * L1, H = P / 2;
  static constexpr int CG = kColGroup;
  static constexpr int NG = H / CG;                       // column groups
  static constexpr int NT = (L1 > 16 ? L1 : 16) * CG;     // one item per thread in each phase
  // element (row, c) of a tile: 16-row blocks are one row of 8 elements apart in
  // FP32, so that the class-parallel accesses of half a warp (two blocks) and
  // the row-parallel ones (two rows) fall on distinct banks
  static constexpr int ROWS = sizeof(T) == 4 ? P + L1 : P;
  __device__ static __forceinline__ int at(int row, int c) {
    return (sizeof(T) == 4 ? row + (row >> 4) : row) * CG + c;
  }
  // offset of row + 16 i from row, and of row 16 b + q from row 16 b
  static constexpr int STEP16 = (sizeof(T) == 4 ? 17 : 16) * CG;
  static constexpr int TILE = ROWS * CG;
  // two tiles (used in turn), the twiddles by class, column 0's spectrum
  static constexpr int TWP = 18;  // pitch of a class's twiddles (16-byte pairs)
  static constexpr size_t SMEM = sizeof(cx<T>) * (2 * TILE + TWP * L1 + P);
  static_assert(H % CG == 0, "column groups tile the half spectrum");
};

// CTAs per SM the register budget is cut for
template <typename T, int L1>
constexpr int col_ctas(size_t smem, int regs32) {
  const int by_regs = 65536 / (ColT<T, L1>::NT * (sizeof(T) == 4 ? regs32 : 232));
  const int by_smem = (int)(232448 / (smem + 1024));
  const int c = by_regs < by_smem ? by_regs : by_smem;
  return c < 1 ? 1 : c;
}

// ---- tensor memory: thread (warp w, lane) owns TMEM lane 32 (w % 4) + lane of the
// CTA's columns; loads and stores are warp-collective
__device__ __forceinline__ uint32_t col_tmem_alloc(uint32_t* slot, uint32_t cols) {
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(slot)),
                 "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  return *slot + ((threadIdx.x & 96u) << 16);
}
__device__ __forceinline__ void col_tmem_free(uint32_t base, uint32_t cols) {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (threadIdx.x < 32)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols)
                 : "memory");
}
// N consecutive columns from column t: a load is issued (ld), its registers may be
// used after the wait (they pass through it, so no use moves above it)
__device__ __forceinline__ void col_tmem_ld(uint32_t t, uint32_t (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {"
               "%0, %1, %2, %3, %4, %5, %6, %7, "
               "%8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]),
                 "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
                 "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(t)
               : "memory");
}
__device__ __forceinline__ void col_tmem_wait_ld(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]),
                 "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]),
                 "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :
               : "memory");
}
__device__ __forceinline__ void col_tmem_st(uint32_t t, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {"
               "%1, %2, %3, %4, %5, %6, %7, %8, "
               "%9, %10, %11, %12, %13, %14, %15, %16};"
               ::"r"(t),
                 "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]),
                 "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                 "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
                 "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
               : "memory");
}
__device__ __forceinline__ void col_tmem_ld(uint32_t t, uint32_t (&r)[32]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {"
               "%0, %1, %2, %3, %4, %5, %6, %7, "
               "%8, %9, %10, %11, %12, %13, %14, %15, "
               "%16, %17, %18, %19, %20, %21, %22, %23, "
               "%24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]),
                 "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
                 "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                 "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
                 "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                 "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
                 "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
               : "r"(t)
               : "memory");
}
__device__ __forceinline__ void col_tmem_wait_ld(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]),
                 "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]),
                 "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]),
                 "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]),
                 "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]),
                 "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]),
                 "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
               :
               : "memory");
}
__device__ __forceinline__ void col_tmem_st(uint32_t t, const uint32_t (&r)[32]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {"
               "%1, %2, %3, %4, %5, %6, %7, %8, "
               "%9, %10, %11, %12, %13, %14, %15, %16, "
               "%17, %18, %19, %20, %21, %22, %23, %24, "
               "%25, %26, %27, %28, %29, %30, %31, %32};"
               ::"r"(t),
                 "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]),
                 "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                 "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
                 "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
                 "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
                 "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
                 "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
                 "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
               : "memory");
}
__device__ __forceinline__ void col_tmem_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

template <typename T, int L1>
__device__ __forceinline__ void load_class_twiddles(cx<T>* stw, const void* tw, int nt) {
  for (int i = threadIdx.x; i < 16 * L1; i += nt) {
    const int c = i >> 4, q = i & 15;
    stw[ColT<T, L1>::TWP * c + q] = __ldg((const cx<T>*)tw + c * q);
  }
}

// slot of ky = -(cls + L1 q) in the class order
template <int L1>
__device__ __forceinline__ int mirror_slot(int cls, int q) {
  constexpr int P = 16 * L1;
  const int km = (P - (cls + L1 * q)) % P;
  return 16 * (km % L1) + km / L1;
}

// rows n2 + 16 i of the window-weighted sky rows (zero outside window and field)
template <typename T, int L1>
__device__ __forceinline__ void load_sky_rows(const ColK& k, const cx<T>* src,
                                              int rb, int n2, cx<T> (&v)[L1]) {
  constexpr int H = 8 * L1;
  const T* __restrict__ wt = (const T*)k.a.wt;
  T w[L1];  // (every load is issued before the first product)
#pragma unroll
  for (int i = 0; i < L1; ++i) {
    const int y = n2 + 16 * i, ya = y - k.margin, row = rb + y;
    const bool ok = (unsigned)ya < (unsigned)k.K && (unsigned)row < (unsigned)k.nx;
    v[i] = ok ? src[(int64_t)row * H] : mkc<T>((T)0, (T)0);
    w[i] = ok ? wt[ya] : (T)0;
  }
#pragma unroll
  for (int i = 0; i < L1; ++i) v[i] = mkc<T>(w[i] * v[i].x, w[i] * v[i].y);
}

__device__ __forceinline__ float2 col_load_past_l1(const float2* p) {
  float2 v;
  asm volatile("ld.global.nc.L1::no_allocate.v2.f32 {%0, %1}, [%2];"
               : "=f"(v.x), "=f"(v.y)
               : "l"(p));
  return v;
}
__device__ __forceinline__ double2 col_load_past_l1(const double2* p) { return __ldg(p); }
// the 16 values of a class: rows 16 cls + q of the (P, H) array h, column col.  PAST_L1:
// lines that are read once leave the L1 to the other loads in flight.  The adjoint takes
// it (FP32; side 384 at 1024^2 x 7 x 3: 305 -> 294 us, side 192 at one module 68.9 ->
// 66.8); the forward, whose sky rows are re-read from L1, does not (291 -> 302).
template <typename T, int L1, bool PAST_L1>
__device__ __forceinline__ void load_class(const cx<T>* h, cx<T> (&v)[16]) {
#pragma unroll
  for (int q = 0; q < 16; ++q)
    v[q] = PAST_L1 ? col_load_past_l1(h + q * (8 * L1)) : __ldg(h + q * (8 * L1));
}
template <typename T, int L1>
__device__ __forceinline__ void tile_to_spectrum(const cx<T>* t, const cx<T>* mytw, cx<T> (&v)[16]) {
#pragma unroll
  for (int q = 0; q < 16; q += 2) {
    cx<T> wa, wb;
    two_twiddles(mytw, q, wa, wb);
    const cx<T> za = t[q * kColGroup], zb = t[(q + 1) * kColGroup];
    v[q] = q ? cmul<T>(za, wa) : za;
    v[q + 1] = cmul<T>(zb, wb);
  }
  Dft<16, false, T>::run(v);
}
template <typename T, int L1>
__device__ __forceinline__ void spectrum_to_tile(cx<T>* t, const cx<T>* mytw, cx<T> (&v)[16]) {
  Dft<16, true, T>::run(v);
#pragma unroll
  for (int q = 0; q < 16; q += 2) {
    cx<T> wa, wb;
    two_twiddles(mytw, q, wa, wb);
    t[q * kColGroup] = q ? cmulc<T>(v[q], wa) : v[q];
    t[(q + 1) * kColGroup] = cmulc<T>(v[q + 1], wb);
  }
}

// Columns of TMEM a CTA of the run kernel takes for mc modules (a power of two).
template <int L1, int D>
constexpr int run_tmem_cols(int mc) {
  int c = 32;
  while (c < 2 * (L1 - D) * mc) c *= 2;
  return c;
}

// Forward columns: sky row spectra -> spectrum of a patch (registers) -> per
// module the PSF product -> rows of the slab.
// D = 0: one patch per CTA, every module.
// D > 0 (FP32): a run of vertically adjacent patches and up to mc modules per
// CTA.  A patch's P rows are P / dx strides; the rows that later patches of the
// run also cover wait in TMEM, per module, so each row of the run's slab is
// written once, summed in patch order.  D = dx / 16: a patch's rows 16 i + q are
// rows 16 (i - D) + q of the next patch, so a thread's pending rows stay with it.
template <typename T, int L1, int D>
__global__ void __launch_bounds__(ColT<T, L1>::NT, col_ctas<T, L1>(ColT<T, L1>::SMEM, 128))
    k_sep_cols_fwd(ColK k) {
  using C = ColT<T, L1>;
  constexpr int P = C::P, H = C::H, CG = C::CG, NT = C::NT, NP = L1 - D;
  static_assert(D == 0 || (sizeof(T) == 4 && (NP == 8 || NP == 16) && NT >= 128),
                "pending rows: 16 or 32 TMEM columns of the four warps of the DFT-L1 phase");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint32_t s_tmem;
  cx<T>* tile = reinterpret_cast<cx<T>*>(smem_raw);
  cx<T>* stw = tile + 2 * C::TILE;
  cx<T>* w0 = stw + C::TWP * L1;
  const int tid = threadIdx.x, c = tid % CG, it = tid / CG;
  int u = blockIdx.x;
  const int cg = u % C::NG;
  u /= C::NG;
  int e, j, i0, R = 1, run = 0;
  if (D == 0) {  // u = e n^2 + patch
    e = sep_div(u, k.n2, k.div_n2);
    const int kp = u - e * k.n2;
    j = sep_div(kp, k.n, k.div_n);
    i0 = kp - j * k.n;
  } else {  // u = (e n + j) nq + run
    const int t = sep_div(u, k.nq, k.div_q);
    run = u - t * k.nq;
    e = sep_div(t, k.n, k.div_n);
    j = t - e * k.n;
    R = k.a.run;
    i0 = run * R;
  }
  const int m0 = D == 0 ? 0 : (int)blockIdx.y * k.mc;
  const int m1 = D == 0 ? k.M : min(k.M, m0 + k.mc);
  const int col = cg * CG + c;
  const bool mid = it < L1;  // this thread holds class it of its column
  const bool tail = it < 16;
  const bool c0 = cg == 0 && c == 0;
  const int kp0 = i0 + k.n * j;
  const cx<T>* hm = (const cx<T>*)k.a.hmain + (16 * it) * H + col;
  auto unit = [&](int m, int s) { return ((int64_t)m * k.n2 + kp0 + s) * k.E + e; };
  const int64_t hstep = (int64_t)k.n2 * k.E * (P * H);  // from module to module
  load_class_twiddles<T, L1>(stw, k.a.tw, NT);
  uint32_t tm = 0;
  if (D > 0) tm = col_tmem_alloc(&s_tmem, run_tmem_cols<L1, D>(k.mc));
  sep_wait();
  const cx<T>* hb = hm + unit(m0, 0) * (P * H);
  cx<T> hv[16];
  if (mid) load_class<T, L1, false>(hb, hv);
  const cx<T>* mytw = stw + C::TWP * it;
  const int mine = C::at(16 * it, c), myrow = C::at(it, c);
  const int height = D == 0 ? P : (R - 1) * k.dx + P;
  int which = 0;  // tile of the next transform
  for (int s = 0; s < R; ++s) {
    const int rb = min((i0 + s) * k.dx, k.sr_max) - k.half - k.margin;
    if (tail) {
      cx<T> v[L1];
      load_sky_rows<T, L1>(k, (const cx<T>*)k.a.rows + ((int64_t)(e * k.n + j) * k.nx) * H + col,
                           rb, it, v);
      Dft<L1, false, T>::run(v);
      cx<T>* t = tile + which * C::TILE + myrow;
#pragma unroll
      for (int i = 0; i < L1; ++i) t[i * C::STEP16] = v[i];
    }
    __syncthreads();
    cx<T> sp[16];
    if (mid) tile_to_spectrum<T, L1>(tile + which * C::TILE + mine, mytw, sp);
    which ^= 1;
    if (cg == 0) {
      if (c0 && mid) {
#pragma unroll
        for (int q = 0; q < 16; ++q) w0[16 * it + q] = sp[q];
      }
      __syncthreads();
    }
    for (int m = m0; m < m1; ++m) {
      cx<T>* buf = tile + which * C::TILE;
      which ^= 1;
      if (mid) {
        cx<T> v[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = cmul<T>(sp[q], hv[q]);
        if (m + 1 < m1) {
          hb += hstep;
          load_class<T, L1, false>(hb, hv);
        } else if (s + 1 < R) {
          hb = hm + unit(m0, s + 1) * (P * H);
          load_class<T, L1, false>(hb, hv);
        }
        if (c0) {
          const cx<T>* be = (const cx<T>*)k.a.hnyq + unit(m, s) * P + 16 * it;
#pragma unroll
          for (int q = 0; q < 16; ++q)
            v[q] = cadd<T>(v[q], cmul<T>(cconj<T>(w0[mirror_slot<L1>(it, q)]), __ldg(be + q)));
        }
        spectrum_to_tile<T, L1>(buf + mine, mytw, v);
      }
      if (m + 1 == m1 && s + 1 == R) sep_trigger();
      __syncthreads();
      if (tail) {
        cx<T> v[L1];
        const cx<T>* t = buf + myrow;
#pragma unroll
        for (int i = 0; i < L1; ++i) v[i] = t[i * C::STEP16];
        Dft<L1, true, T>::run(v);
        const int64_t pl = (int64_t)m * k.E + e;
        const int y0 = s * k.dx + it;  // the thread's first row within the slab
        cx<T>* dst = (cx<T>*)k.a.slab +
                     (((pl * k.n + j) * k.nq + (D == 0 ? i0 : run)) * height + y0) * H + col;
        int leave = L1;
        if constexpr (D > 0) {
          uint32_t pend[2 * NP];  // the pending rows of this module
          const uint32_t tp = tm + (uint32_t)(2 * NP * (m - m0));
          if (s > 0) {
            col_tmem_ld(tp, pend);
            col_tmem_wait_ld(pend);
#pragma unroll
            for (int i = 0; i < NP; ++i)
              v[i] = mkc<T>(__uint_as_float(pend[2 * i]) + v[i].x,
                            __uint_as_float(pend[2 * i + 1]) + v[i].y);
          }
          if (s + 1 < R) {
            leave = D;
#pragma unroll
            for (int i = 0; i < NP; ++i) {
              pend[2 * i] = __float_as_uint((float)v[D + i].x);
              pend[2 * i + 1] = __float_as_uint((float)v[D + i].y);
            }
            col_tmem_st(tp, pend);
          }
        }
#pragma unroll
        for (int i = 0; i < L1; ++i)
          if (i < leave && (unsigned)(rb + 16 * i + it) < (unsigned)k.nx) dst[16 * i * H] = v[i];
        if (D > 0) col_tmem_wait_st();
      }
    }
  }
  if (D > 0) col_tmem_free(s_tmem, run_tmem_cols<L1, D>(k.mc));
}

// Asynchronous 16-byte global -> shared copy (ok false: zeros, nothing read).
__device__ __forceinline__ void col_copy16(void* dst, const void* src, bool ok) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(ok ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void col_copy_wait() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
}
// P rows of a patch (rows rb ... of the image, zeros outside the field), CG columns -> tile
template <typename T, int L1>
__device__ __forceinline__ void col_fetch_rows(cx<T>* tile, const cx<T>* src, int rb, int nx,
                                               int tid) {
  using C = ColT<T, L1>;
  constexpr int EL = 16 / (int)sizeof(cx<T>), RB = C::CG / EL;  // values a chunk, chunks a row
#pragma unroll
  for (int i = 0; i < (C::P * RB + C::NT - 1) / C::NT; ++i) {
    const int ch = tid + i * C::NT;
    if ((C::P * RB) % C::NT && ch >= C::P * RB) break;
    const int row = ch / RB, part = ch % RB, g = rb + row;
    const bool ok = (unsigned)g < (unsigned)nx;
    col_copy16(tile + C::at(row, part * EL), src + (int64_t)(ok ? g : 0) * C::H + part * EL, ok);
  }
}

// class it of patch u's sums between chunks, behind the gradient slabs
template <typename T, int L1>
__device__ __forceinline__ cx<T>* col_sums(const ColK& k, int u, int it) {
  constexpr int P = 16 * L1, H = P / 2;
  return (cx<T>*)k.a.slab + (int64_t)k.E * k.n2 * k.K * H + ((int64_t)u * P + 16 * it) * H;
}

// Adjoint columns of one patch: per module the row spectra of the patch's rows
// -> spectrum -> conjugate PSF product, summed over modules in registers in
// module order; the sum's inverse columns, weighted by the window rows, to the
// patch's gradient slab.  The next module's rows arrive by cp.async in the other
// tile, its PSF spectrum in registers, while this module is transformed.  CHUNK: the modules
// come in several launches, and the sums wait behind the gradient slabs between them.
template <typename T, int L1, bool CHUNK>
__global__ void __launch_bounds__(ColT<T, L1>::NT, col_ctas<T, L1>(ColT<T, L1>::SMEM, 128))
    k_sep_cols_adj(ColK k) {
  using C = ColT<T, L1>;
  constexpr int P = C::P, H = C::H, CG = C::CG, NT = C::NT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cx<T>* tile = reinterpret_cast<cx<T>*>(smem_raw);
  cx<T>* stw = tile + 2 * C::TILE;
  cx<T>* w0 = stw + C::TWP * L1;
  const int tid = threadIdx.x, c = tid % CG, it = tid / CG;
  int u = blockIdx.x;
  const int cg = u % C::NG;
  u /= C::NG;
  const int e = sep_div(u, k.n2, k.div_n2), kp = u - e * k.n2;
  const int j = sep_div(kp, k.n, k.div_n), i0 = kp - j * k.n;
  const int rb = min(i0 * k.dx, k.sr_max) - k.half - k.margin;
  const int col = cg * CG + c;
  const bool mid = it < L1, tail = it < 16;
  const bool c0 = cg == 0 && c == 0;
  const cx<T>* hb =
      (const cx<T>*)k.a.hmain + ((int64_t)kp * k.E + e) * (P * H) + (16 * it) * H + col;
  const int64_t hstep = (int64_t)k.n2 * k.E * (P * H);
  const cx<T>* src = (const cx<T>*)k.a.rows + ((int64_t)(e * k.n + j) * k.nx) * H + cg * CG;
  const int64_t rstep = (int64_t)k.E * k.n * k.nx * H;
  load_class_twiddles<T, L1>(stw, k.a.tw, NT);
  cx<T> hv[16];
  if (mid) load_class<T, L1, true>(hb, hv);
  sep_wait();
  col_fetch_rows<T, L1>(tile, src, rb, k.nx, tid);
  const cx<T>* mytw = stw + C::TWP * it;
  const int mine = C::at(16 * it, c), myrow = C::at(it, c);
  cx<T> acc[16];
#pragma unroll
  for (int q = 0; q < 16; ++q) acc[q] = mkc<T>((T)0, (T)0);
  if (CHUNK && (k.a.run & SEP_RESUME) && mid) {
    const cx<T>* sums = col_sums<T, L1>(k, u, it) + col;
#pragma unroll
    for (int q = 0; q < 16; ++q) acc[q] = sums[q * H];
  }
  for (int m = 0; m < k.M; ++m) {
    cx<T>* buf = tile + ((m & 1) ? C::TILE : 0);
    col_copy_wait();
    __syncthreads();  // module m's rows are here, and the other tile has been read
    src += rstep;
    if (m + 1 < k.M)
      col_fetch_rows<T, L1>(tile + ((m & 1) ? 0 : C::TILE), src, rb, k.nx, tid);
    if (tail) {  // in place: rows it + 16 i of one column
      cx<T> v[L1];
      cx<T>* t = buf + myrow;
#pragma unroll
      for (int i = 0; i < L1; ++i) v[i] = t[i * C::STEP16];
      Dft<L1, false, T>::run(v);
#pragma unroll
      for (int i = 0; i < L1; ++i) t[i * C::STEP16] = v[i];
    }
    __syncthreads();
    if (mid) {
      cx<T> v[16];
      tile_to_spectrum<T, L1>(buf + mine, mytw, v);
#pragma unroll
      for (int q = 0; q < 16; ++q) acc[q] = cmulc_add(v[q], hv[q], acc[q]);
      hb += hstep;
      if (m + 1 < k.M) load_class<T, L1, true>(hb, hv);
      if (c0) {
#pragma unroll
        for (int q = 0; q < 16; ++q) w0[16 * it + q] = v[q];
      }
    }
    if (cg == 0) {
      __syncthreads();
      if (c0 && mid) {
        const cx<T>* be =
            (const cx<T>*)k.a.hnyq + (((int64_t)m * k.n2 + kp) * k.E + e) * P + 16 * it;
#pragma unroll
        for (int q = 0; q < 16; ++q)
          acc[q] = cmulc_add(cconj<T>(w0[mirror_slot<L1>(it, q)]), __ldg(be + q), acc[q]);
      }
    }
  }
  sep_trigger();
  if (CHUNK && (k.a.run & SEP_PASS_ON)) {  // more module chunks to come
    if (mid) {
      cx<T>* sums = col_sums<T, L1>(k, u, it) + col;
#pragma unroll
      for (int q = 0; q < 16; ++q) sums[q * H] = acc[q];
    }
    return;
  }
  cx<T>* buf = tile + ((k.M & 1) ? C::TILE : 0);
  if (mid) spectrum_to_tile<T, L1>(buf + mine, mytw, acc);
  __syncthreads();
  if (tail) {
    const T* __restrict__ wt = (const T*)k.a.wt;
    cx<T>* dst = (cx<T>*)k.a.slab + (int64_t)u * k.K * H + col;
    cx<T> v[L1];
    const cx<T>* t = buf + myrow;
#pragma unroll
    for (int i = 0; i < L1; ++i) v[i] = t[i * C::STEP16];
    Dft<L1, true, T>::run(v);
#pragma unroll
    for (int i = 0; i < L1; ++i) {
      const int ya = 16 * i + it - k.margin;
      if (ya >= 0 && ya < k.K) {
        const T w = wt[ya];
        dst[(int64_t)ya * H] = mkc<T>(w * v[i].x, w * v[i].y);
      }
    }
  }
}

// Strides of 16 rows from patch to patch (dx / 16) that the run kernel covers for
// a side of 16 L1: P = 3 dx, the margin rule of the demo geometries (0: none).
template <typename T, int L1>
constexpr int run_shift() {
  return sizeof(T) == 4 && (L1 == 12 || L1 == 24) ? L1 / 3 : 0;
}

// Modules per CTA of the run kernel: as many as the TMEM columns of the CTAs that share
// an SM hold.
template <int L1, int D>
int run_modules(int M, int per_sm) {
  return std::min(M, std::max(1, 512 / per_sm / (2 * (L1 - D))));
}

// Waves of CTAs of the run kernel for runs of r patches.
template <typename T, int L1>
double run_waves(const Geom& g, int r) {
  const int per_sm = col_ctas<T, L1>(ColT<T, L1>::SMEM, 128);
  const int mc = run_modules<L1, run_shift<T, L1>()>(g.M, per_sm);
  const double ctas = (double)g.E * g.n * (g.n / r) * ColT<T, L1>::NG * ((g.M + mc - 1) / mc);
  return ctas / ((double)sm_count() * per_sm);
}

template <typename T, int L1>
int dispatch_cols(const Geom& g, SepColsKind kind, const SepCols& a, bool pdl, cudaStream_t s) {
  using C = ColT<T, L1>;
  ColK k{};
  k.a = a;
  k.M = g.M;
  k.E = g.E;
  k.nx = g.nx;
  k.n = g.n;
  k.n2 = g.n * g.n;
  k.dx = g.dx;
  k.half = g.half;
  k.margin = g.margin;
  k.sr_max = g.sr_max;
  k.K = g.K;
  k.nq = kind == SEP_COLS_FWD ? g.n / a.run : g.n;
  const int64_t patches = (int64_t)g.E * k.n2;
  const int64_t grid = (a.run > 1 && kind == SEP_COLS_FWD ? (int64_t)g.E * g.n * k.nq : patches) *
                       C::NG;
  if (grid > 0x7fffffffLL) {
    set_error("separable columns: too many patches for one launch");
    return JUBIK_ERR_UNSUPPORTED;
  }
  k.div_n2 = mulhi_divisor(k.n2, patches + 1);
  k.div_n = mulhi_divisor(g.n, patches + 1);
  k.div_q = mulhi_divisor(k.nq, grid + 1);
  dim3 gd((unsigned)grid);
  int per_sm = 1;
  if (kind == SEP_COLS_ADJ && (a.run & (SEP_RESUME | SEP_PASS_ON))) {
    static SepKernelCache cache;
    auto kern = k_sep_cols_adj<T, L1, true>;
    JUBIK_TRY(cache.prepare((const void*)kern, C::NT, C::SMEM, &per_sm));
    return sep_launch(kern, gd, C::NT, C::SMEM, pdl, s, "k_sep_cols_adj (chunk)", k);
  }
  if (kind == SEP_COLS_ADJ) {
    static SepKernelCache cache;
    auto kern = k_sep_cols_adj<T, L1, false>;
    JUBIK_TRY(cache.prepare((const void*)kern, C::NT, C::SMEM, &per_sm));
    return sep_launch(kern, gd, C::NT, C::SMEM, pdl, s, "k_sep_cols_adj", k);
  }
  if (a.run > 1) {
    constexpr int D = run_shift<T, L1>();
    if constexpr (D > 0) {
      static SepKernelCache cache;
      auto kern = k_sep_cols_fwd<T, L1, D>;
      JUBIK_TRY(cache.prepare((const void*)kern, C::NT, C::SMEM, &per_sm));
      k.mc = run_modules<L1, D>(g.M, per_sm);
      gd.y = (unsigned)((g.M + k.mc - 1) / k.mc);
      return sep_launch(kern, gd, C::NT, C::SMEM, pdl, s, "k_sep_cols_fwd (runs)", k);
    }
    set_error("separable columns: no runs of patches at P=%d", g.P);
    return JUBIK_ERR_UNSUPPORTED;
  }
  static SepKernelCache cache;
  auto kern = k_sep_cols_fwd<T, L1, 0>;
  JUBIK_TRY(cache.prepare((const void*)kern, C::NT, C::SMEM, &per_sm));
  return sep_launch(kern, gd, C::NT, C::SMEM, pdl, s, "k_sep_cols_fwd", k);
}

}  // namespace

template <typename T>
int sep_cols_t(const Geom& g, SepColsKind kind, const SepCols& a, bool pdl, cudaStream_t s) {
  switch (g.P) {
    case 160: return dispatch_cols<T, 10>(g, kind, a, pdl, s);
    case 192: return dispatch_cols<T, 12>(g, kind, a, pdl, s);
    case 256: return dispatch_cols<T, 16>(g, kind, a, pdl, s);
    case 320: return dispatch_cols<T, 20>(g, kind, a, pdl, s);
    case 384: return dispatch_cols<T, 24>(g, kind, a, pdl, s);
    case 512: return dispatch_cols<T, 32>(g, kind, a, pdl, s);
    default: break;
  }
  set_error("separable columns do not cover P=%d", g.P);
  return JUBIK_ERR_UNSUPPORTED;
}

}  // namespace jubik
