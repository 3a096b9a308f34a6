// Row kernels of the separable response (see sep.h).
//
// A CTA takes one or more pairs of image rows (2t, 2t + 1) of one plane with
// all n windows (patch columns) that cut them.  The two real rows of a pair
// travel as the real and imaginary part of one complex sequence per window.
//   inverse half: slabs -> row spectra of the pair (sum over the slabs that
//     cover the row, in order) -> inverse transforms -> overlap-add over the
//     windows in shared memory (window order, two words) -> image rows;
//   pixels: likelihood, metric weights, readout, gradient, ...;
//   forward half: image rows -> windows -> transforms -> row spectra.
// Both halves run in one kernel for the likelihood and the metric, so the image
// of expected counts is never stored.
//
// Each transform of side P = 16 L1 is a two-phase four-step in place: slots
// 16 cls + q lie at 17 cls + q (the odd class pitch spreads both the
// class-parallel and the slot-parallel accesses over the banks).  A warp takes two
// sequences through all of its phases -- load and join of the two rows' spectra,
// DFT-L1 (16 classes x 2 sequences: one per lane), DFT-16; and back -- with warp
// barriers only; the CTA meets twice per item, before and after the overlap-add.
// The kernels are bound by the latency of the spectrum loads and by instruction
// issue; warps that drift apart overlap the one with the other.  At 1024^2 x 7 x 3
// the likelihood's rows move 858 MB in 287 us (3.0 TB/s), issue slots 62 % busy at 512^2.
#include "likelihood.cuh"
#include "sep_dev.cuh"

namespace jubik {
namespace {

struct RowK {
  SepRows a;
  int mode;
  int nx, ny, n, dx, half, margin, sr_max, sc_max, K;
  int nslab, step, height;   // slabs of a patch column: start every step rows, height rows
  int late;                  // rows the last slab starts before its stride (clamped windows)
  int few;                   // at most 4 windows cover a column, all in buf, none clamped
  int seqs;                  // sequences (row pair x window) in shared memory at once
  int rp;                    // row pairs per item
  int per;                   // items per plane
  int grid_items;            // items of the whole image
  int item0, items;          // this launch's items: item0 .. items - 1
  int base;                  // the multiple of the grid before item0
  uint32_t mul_dx, mul_step;  // floor(u / d) = high word of u mul (row_div)
  uint32_t div_per;
  float scale32[2];  // the factor's two words
  double scale64[2];
};
template <typename T> __device__ __forceinline__ T row_scale(const RowK& k, int word);
template <> __device__ __forceinline__ float row_scale<float>(const RowK& k, int word) {
  return k.scale32[word];
}
template <> __device__ __forceinline__ double row_scale<double>(const RowK& k, int word) {
  return k.scale64[word];
}

// Sequences (row pair x window) a CTA holds at once: 16, or as many as fit beside
// the image rows of a wide field (row_seqs).
constexpr int kRowSeqs = 16;

template <int L1>
constexpr int row_pitch() { return 17 * L1 + (L1 % 16 == 0 ? 8 : 0); }
constexpr int kRowThreads = 16 * kRowSeqs;  // two sequences a warp
// CTAs per SM the register budget is cut for: 80 registers (FP32), 128 for the
// long DFT-L1 of P >= 320 and for FP64, 255 for both
template <typename T, int L1>
constexpr int row_ctas() { return sizeof(T) == 4 ? (L1 <= 16 ? 3 : 2) : (L1 <= 16 ? 2 : 1); }
constexpr int kRowTw = 18;  // pitch of a class's twiddles (16-byte pairs)

// bytes of dynamic shared memory: sequences, twiddles by class, image rows (and,
// with more windows than sequences, the overlap-add's compensation), windows by column
template <typename T, int L1>
size_t row_smem(int n, int ny, int rp, int most) {
  const size_t seqs = (size_t)std::min(most, n * rp) * row_pitch<L1>();
  const size_t lines = (size_t)rp * ny * (n > most ? 2 : 1);
  const size_t red = 2 * sizeof(double) * kRowThreads;  // the block sums reuse seqs
  return std::max(sizeof(cx<T>) * seqs, red) + sizeof(cx<T>) * (lines + kRowTw * L1) +
         sizeof(uint32_t) * ny;
}
inline int row_pairs(int n, int nx, int most) {  // row pairs of an item
  return std::min(std::max(1, most / n), (nx + 1) / 2);
}
// the most sequences (of 16, 8, 4, 2) that fit beside the rows of this field; 0: none
template <typename T, int L1>
int row_seqs(const Geom& g) {
  for (int most = kRowSeqs; most >= 2; most /= 2)
    if (row_smem<T, L1>(g.n, g.ny, row_pairs(g.n, g.nx, most), most) + 1024 <=
        (size_t)max_smem_optin())
      return most;
  return 0;
}

// floor(u / d) for 0 <= u by the multiply-high constant of d >= 2 (mulhi_divisor)
__device__ __forceinline__ int row_div(int u, uint32_t mul) { return (int)__umulhi((uint32_t)u, mul); }
__device__ __forceinline__ int row_slot(int z) { return (z >> 4) * 17 + (z & 15); }

// Writes p = a + i b at kx = lane + 32 t and conj m, m = a - i b, at P - kx of the pair's
// sequence (kx = 0: the packed real kx = 0 and kx = P / 2 values of a and b).
template <typename T, int L1>
__device__ __forceinline__ void row_store(cx<T> p, cx<T> m, const cx<T>& a, const cx<T>& b, int t,
                                          cx<T>* wp, cx<T>* wm, int lane) {
  const bool dc = t == 0 && lane == 0;
  wp[34 * t] = dc ? mkc<T>(a.x, b.x) : p;
  (dc ? wp + row_slot(8 * L1) : wm - 34 * t)[0] = dc ? mkc<T>(a.y, b.y) : cconj<T>(m);
}
// Joins the two rows' values.
template <typename T, int L1>
__device__ __forceinline__ void row_join(const cx<T> (&v)[2], int t, cx<T>* wp, cx<T>* wm,
                                         int lane) {
  const cx<T> ib = cmul_i<T>(v[1]);
  row_store<T, L1>(cadd<T>(v[0], ib), csub<T>(v[0], ib), v[0], v[1], t, wp, wm, lane);
}
// The same for sums v + lo of two words.
template <typename T, int L1>
__device__ __forceinline__ void row_join2(const cx<T> (&v)[2], const cx<T> (&lo)[2], int t,
                                          cx<T>* wp, cx<T>* wm, int lane) {
  const cx<T> ib = cmul_i<T>(v[1]), il = cmul_i<T>(lo[1]);
  cx<T> p, pe, m, me;
  two_sum(v[0], ib, p, pe);
  two_sum(v[0], mkc<T>(-ib.x, -ib.y), m, me);
  p = padd(p, padd(pe, padd(lo[0], il)));
  m = padd(m, padd(me, psub(lo[0], il)));
  row_store<T, L1>(p, m, padd(v[0], lo[0]), padd(v[1], lo[1]), t, wp, wm, lane);
}

// Spectra of a row pair in one window: the sum of up to N slabs, in FP32 in two words (in
// FP64 the two words cost 14 % of a pass and changed its error by 0.3 %).  The loads
// of three steps are issued before the first sum: with one loop for up to three slabs the
// compiler interleaved loads and sums, and the likelihood's rows took 331 us at
// 1024^2 x 7 x 3 and 381 at side 384, then 272 and 268; with two words 289 and 280.
template <typename T, int L1, int N>
__device__ __forceinline__ void row_load(const cx<T>* p, const int (&o)[2][3], const int (&m)[2],
                                         cx<T>* wp, cx<T>* wm, int lane) {
  constexpr int H = 8 * L1, STEPS = (H + 31) / 32, G = sizeof(T) == 4 ? 3 : 1;
  constexpr bool TWO = N > 1 && sizeof(T) == 4;
#pragma unroll
  for (int t0 = 0; t0 < STEPS; t0 += G) {
    cx<T> z[G][2][N];
#pragma unroll
    for (int t = t0; t < t0 + G && t < STEPS; ++t) {
      const bool in = H % 32 == 0 || lane + 32 * t < H;
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int u = 0; u < N; ++u)
          z[t - t0][b][u] =
              in && u < m[b] ? p[o[b][u] + 32 * t] : mkc<T>((T)0, (T)0);
    }
#pragma unroll
    for (int t = t0; t < t0 + G && t < STEPS; ++t) {
      if (H % 32 && lane + 32 * t >= H) break;
      cx<T> v[2], lo[2];
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        v[b] = z[t - t0][b][0];
        lo[b] = mkc<T>((T)0, (T)0);
#pragma unroll
        for (int u = 1; u < N; ++u) {
          if (TWO) {
            cx<T> e;
            two_sum(v[b], z[t - t0][b][u], v[b], e);
            lo[b] = u == 1 ? e : padd(lo[b], e);
          } else {
            v[b] = cadd<T>(v[b], z[t - t0][b][u]);
          }
        }
      }
      if (TWO)
        row_join2<T, L1>(v, lo, t, wp, wm, lane);
      else
        row_join<T, L1>(v, t, wp, wm, lane);
    }
  }
}

// s + e = s0 + e0 + w z up to the rounding of the low words
template <typename T>
__device__ __forceinline__ void add_weighted(T w, cx<T> z, cx<T> s0, cx<T> e0, cx<T>& s, cx<T>& e) {
  const cx<T> p = pmul(both<T>(w), z);
  const cx<T> pe = pfma(both<T>(w), z, mkc<T>(-p.x, -p.y));
  cx<T> er;
  two_sum(s0, p, s, er);
  e = padd(e0, padd(er, pe));
}

// DFT-L1 of class `ca` of a sequence, in place
template <typename T, int L1, bool INV>
__device__ __forceinline__ void row_dft_l1(cx<T>* seq, int ca) {
  cx<T>* row = seq + ca;
  cx<T> v[L1];
#pragma unroll
  for (int i = 0; i < L1; ++i) v[i] = row[17 * i];
  Dft<L1, INV, T>::run(v);
#pragma unroll
  for (int i = 0; i < L1; ++i) row[17 * i] = v[i];
}

// MODE: what happens to the pixels (SEP_IMAGE also serves SEP_READOUT and
// SEP_WEIGHTS, by a.mode; SEP_COT also SEP_COT_READOUT).  FWD: transform the rows
// that result.
template <typename T, int L1, int MODE, bool FWD>
__global__ void __launch_bounds__(kRowThreads, row_ctas<T, L1>()) k_sep_rows(RowK k) {
  constexpr int P = 16 * L1, H = P / 2, WP = row_pitch<L1>();
  constexpr bool INV = MODE != SEP_SKY && MODE != SEP_COT, GRAD = MODE == SEP_GRAD;
  // sequences whose DFT-16 items a warp runs at once (L1 lanes each)
  constexpr int SEQ16 = 2 * L1 <= 32 ? 2 : 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const SepRows& a = k.a;
  const int n = k.n, ny = k.ny, nx = k.nx;
  const int nsq = min(k.seqs, n * k.rp);
  const size_t seq_bytes = max(sizeof(cx<T>) * (size_t)(nsq * WP), 2 * sizeof(double) * kRowThreads);
  cx<T>* buf = reinterpret_cast<cx<T>*>(smem_raw);
  cx<T>* stw = reinterpret_cast<cx<T>*>(smem_raw + seq_bytes);
  cx<T>* line = stw + kRowTw * L1;
  cx<T>* comp = line + (size_t)k.rp * ny;  // n > k.seqs only
  uint32_t* xwin = reinterpret_cast<uint32_t*>(line + (size_t)k.rp * ny * (n > k.seqs ? 2 : 1));
  const int tid = threadIdx.x, NT = blockDim.x, lane = tid & 31;
  const int q0 = 2 * (tid >> 5);          // this warp's sequences: q0, q0 + 1
  const int cls = lane % L1, sub = lane / L1;  // this lane's DFT-16 item
  // slots of kx = lane and of kx = P - lane (32 further on: 34 slots)
  const int slot_p = row_slot(lane), slot_m = row_slot(P - lane);
  const T* __restrict__ wt = (const T*)a.wt;
  const T* __restrict__ eps = (const T*)a.eps;
  const int off = GRAD ? k.margin : 0;
  const int base_c = -k.half - k.margin + off;
  const int wx = GRAD ? k.K : P;  // window columns the overlap-add takes
  {
    const cx<T>* tw = (const cx<T>*)a.tw;
    for (int i = tid; i < 16 * L1; i += NT) {
      const int cc = i >> 4, q = i & 15;
      stw[kRowTw * cc + q] = __ldg(tw + cc * q);
    }
  }
  if (INV) {
    // the windows that cover column x: the first one and their count
    for (int x = tid; x < ny; x += NT) {
      const int d = x - base_c, under = d - wx + 1;
      int hi = min(n - 1, row_div(d, k.mul_dx));
      // a last window that starts early (clamped) may cover x too
      if (hi + 1 == n - 1 && k.sc_max <= d) ++hi;
      const int lo = under <= 0 ? 0 : row_div(under + k.dx - 1, k.mul_dx);
      const uint32_t cw = hi >= lo ? (uint32_t)(hi - lo + 1) : 0u;
      const int xi = d - lo * k.dx;  // x within window lo
      // few: place of x in window lo, count, xi; else: lo, count
      if (k.few)
        xwin[x] = cw ? ((uint32_t)xi << 20 | cw << 16 | (uint32_t)(lo * WP + xi + off)) : 0u;
      else
        xwin[x] = cw ? ((uint32_t)lo << 16 | cw) : 0u;
    }
  }
  sep_wait();
  __syncthreads();
  const cx<T>* mytw = stw + kRowTw * cls;
  const T scale = row_scale<T>(k, 0), scale_lo = row_scale<T>(k, 1);
  Kahan2<T> s_lam, s_dlog;
  const int nchunk = (n * k.rp + k.seqs - 1) / k.seqs;  // > 1 only when rp == 1
  if (MODE == SEP_LIKE && a.state && a.plane0) {  // the sums of the chunks before
    const cx<T>* st = (const cx<T>*)a.state + 4 * ((int64_t)blockIdx.x * NT + tid);
    s_lam.s = st[0];
    s_lam.nc = st[1];
    s_dlog.s = st[2];
    s_dlog.nc = st[3];
  }
  // the first item of this launch that is this CTA's in the whole image
  int item = k.base + blockIdx.x;
  if (item < k.item0) item += gridDim.x;

  for (; item < k.items; item += gridDim.x) {
    const int pl = sep_div(item, k.per, k.div_per);
    const int t0 = (item - pl * k.per) * k.rp;  // first row pair
    if (INV) {
      // ---- slabs -> image rows
      for (int ch = 0; ch < nchunk; ++ch) {
        const int j0 = ch * k.seqs, jn = min(k.seqs, n - j0);  // windows j0 .. j0 + jn - 1
        const int cnt = jn * k.rp;                                 // sequences in buf
        const int hs = k.height * H;
        // the slabs that cover the pair's rows, in order (a row beyond the field: none):
        // their number and the row's offset in each
        int lo_i[2], m[2], o[2][3], had = -1;
#pragma unroll 1
        for (int s = q0; s < q0 + 2 && s < cnt; ++s) {
          const int r = k.rp == 1 ? 0 : s / jn, j = j0 + s - r * jn;
          const int row0 = 2 * (t0 + r);
          if (r != had) {
            had = r;
#pragma unroll
            for (int b = 0; b < 2; ++b) {
              const int d = row0 + b - base_c, under = d - k.height + 1;
              int hi = min(k.nslab - 1, row_div(d, k.mul_step));
              if (hi + 1 == k.nslab - 1 && k.nslab * k.step - k.step - k.late <= d) ++hi;
              lo_i[b] = under <= 0 ? 0 : row_div(under + k.step - 1, k.mul_step);
              m[b] = row0 + b < nx ? hi - lo_i[b] + 1 : 0;
#pragma unroll
              for (int u = 0; u < 3; ++u) {
                const int i = lo_i[b] + u;
                o[b][u] = i * hs + (d - i * k.step + (i == k.nslab - 1 ? k.late : 0)) * H;
              }
            }
          }
          const cx<T>* p = (const cx<T>*)a.slab + ((int64_t)pl * n + j) * hs * k.nslab + lane;
          cx<T>* wp = buf + s * WP + slot_p;
          cx<T>* wm = buf + s * WP + slot_m;
          const int most = max(m[0], m[1]);
          if (most <= 1) {
            row_load<T, L1, 1>(p, o, m, wp, wm, lane);
          } else if (most == 2) {
            row_load<T, L1, 2>(p, o, m, wp, wm, lane);
          } else if (most == 3) {
            row_load<T, L1, 3>(p, o, m, wp, wm, lane);
          } else {  // margins beyond half a stride: more slabs
            const int late = k.late * H;
#pragma unroll 1
            for (int t = 0; t < (H + 31) / 32; ++t) {
              if (H % 32 && lane + 32 * t >= H) break;
              cx<T> v[2], lo[2];
#pragma unroll
              for (int b = 0; b < 2; ++b) {
                v[b] = lo[b] = mkc<T>((T)0, (T)0);
                const int step = hs - k.step * H, first = o[b][0];
#pragma unroll 4
                for (int u = 0; u < m[b]; ++u) {
                  cx<T> e;
                  two_sum(v[b], p[first + u * step + 32 * t +
                                  (u && lo_i[b] + u == k.nslab - 1 ? late : 0)], v[b], e);
                  lo[b] = padd(lo[b], e);
                }
              }
              row_join2<T, L1>(v, lo, t, wp, wm, lane);
            }
          }
        }
        __syncwarp();
        if (q0 + (lane >> 4) < cnt) row_dft_l1<T, L1, true>(buf + (q0 + (lane >> 4)) * WP, lane & 15);
        __syncwarp();
#pragma unroll 1
        for (int h = 0; h < 2; h += SEQ16) {  // DFT-16 -> natural order
          const int s = q0 + h + sub;
          const bool on = sub < SEQ16 && s < cnt;
          cx<T> v[16];
          if (on) {
            const cx<T>* src = buf + s * WP + 17 * cls;
#pragma unroll
            for (int q = 0; q < 16; q += 2) {
              cx<T> wa, wb;
              two_twiddles(mytw, q, wa, wb);
              v[q] = q ? cmulc<T>(src[q], wa) : src[q];
              v[q + 1] = cmulc<T>(src[q + 1], wb);
            }
            Dft<16, true, T>::run(v);
          }
          __syncwarp();  // in place: every lane has read
          if (on) {
            cx<T>* dst = buf + s * WP + cls;
#pragma unroll
            for (int q = 0; q < 16; ++q) dst[L1 * q] = v[q];
          }
        }
        __syncthreads();
        // overlap-add over the windows, in window order, and the pixels
        const bool last = ch == nchunk - 1;
        for (int r = 0; r < k.rp; ++r) {
          const int row0 = 2 * (t0 + r);
          if (row0 >= nx) break;
          const int64_t px0 = ((int64_t)pl * nx + row0) * ny;
          const bool two = row0 + 1 < nx;
          const cx<T>* wbuf = buf + (r * jn) * WP;
          constexpr int U = 4;  // columns whose pixel inputs are loaded together
          for (int xb = tid; xb < ny; xb += U * NT) {
            T f[U][2];
            int32_t ix[U][2];
            if (MODE == SEP_GRAD) {
#pragma unroll
              for (int u = 0; u < U; ++u) f[u][0] = f[u][1] = (T)1;
            } else {
#pragma unroll
              for (int u = 0; u < U; ++u)
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                  const int x = xb + u * NT;
                  const int64_t p = px0 + (int64_t)b * ny + x;
                  f[u][b] = (T)1;
                  ix[u][b] = -1;
                  if (last && x < ny && (b == 0 || two)) {
                    if (MODE == SEP_LIKE) ix[u][b] = a.dimg[p];
                    if (MODE == SEP_METRIC) f[u][b] = ((const T*)a.wts)[p];
                    if (MODE == SEP_IMAGE && k.mode != SEP_IMAGE) ix[u][b] = a.ridx[p];
                    if (MODE != SEP_METRIC && eps && (MODE == SEP_LIKE || k.mode != SEP_IMAGE))
                      f[u][b] = eps[p];
                  }
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
              const int x = xb + u * NT;
              if (x >= ny) break;
              const uint32_t e = xwin[x];
              cx<T> sum, rest;  // the two words of the sum over the windows
              if (k.few) {
                // up to four windows' values, in window order
                const cx<T>* w = wbuf + (e & 0xffffu);
                const int cw = (int)(e >> 16) & 15, S = WP - k.dx;
                const cx<T> z = mkc<T>((T)0, (T)0);
                const cx<T> z0 = cw > 0 ? w[0] : z, z1 = cw > 1 ? w[S] : z;
                const cx<T> z2 = cw > 2 ? w[2 * S] : z;
                if (GRAD) {  // the windows' column weights
                  const T* wx0 = wt + (e >> 20);
                  const T g0 = cw > 0 ? wx0[0] : (T)0, g1 = cw > 1 ? wx0[-k.dx] : (T)0;
                  const T g2 = cw > 2 ? wx0[-2 * k.dx] : (T)0;
                  add_weighted<T>(g0, z0, z, z, sum, rest);
                  add_weighted<T>(g1, z1, sum, rest, sum, rest);
                  add_weighted<T>(g2, z2, sum, rest, sum, rest);
                  if (cw > 3)
                    add_weighted<T>(wt[(int)(e >> 20) - 3 * k.dx], w[3 * S], sum, rest, sum, rest);
                } else {
                  cx<T> er;
                  two_sum(z0, z1, sum, rest);
                  two_sum(sum, z2, sum, er);
                  rest = padd(rest, er);
                  if (cw > 3) {
                    two_sum(sum, w[3 * S], sum, er);
                    rest = padd(rest, er);
                  }
                }
              } else {
                int j = (int)(e >> 16), jend = j + (int)(e & 0xffffu);
                j = max(j, j0);
                jend = min(jend, j0 + jn);
                sum = rest = mkc<T>((T)0, (T)0);
                if (ch > 0) {
                  sum = line[x];
                  rest = comp[x];
                }
                const cx<T>* w = wbuf + (j - j0) * WP + x + off - base_c;
                for (int st = j * k.dx; j < jend; ++j, st += k.dx, w += WP) {
                  const int s0 = min(st, k.sc_max);
                  const cx<T> z = w[-s0];
                  if (GRAD) {
                    add_weighted<T>(wt[x - base_c - s0], z, sum, rest, sum, rest);
                  } else {
                    cx<T> er;
                    two_sum(sum, z, sum, er);
                    rest = padd(rest, er);
                  }
                }
                if (!last) {
                  line[x] = sum;
                  comp[x] = rest;
                  continue;
                }
              }
              // the scaled sum in two words: v, and what v lacks
              const cx<T> v = pmul(both<T>(scale), sum);
              const cx<T> vl = pfma(both<T>(scale), rest,
                                    pfma(both<T>(scale_lo), sum,
                                         pfma(both<T>(scale), sum, mkc<T>(-v.x, -v.y))));
              const int64_t p = px0 + x;
              if (MODE == SEP_LIKE) {
                cx<T> wgt, res;
                poisson_px2<T>(v, vl, mkc<T>(f[u][0], f[u][1]), ix[u], wgt, res, s_lam, s_dlog);
                __stcs((T*)a.wts + p, wgt.x);
                if (two) __stcs((T*)a.wts + p + ny, wgt.y);
                if (FWD) line[r * ny + x] = pmul(both<T>((T)0.5), res);
              } else {
                const cx<T> fv = mkc<T>(f[u][0], f[u][1]);
                // (factor) (v + vl), rounded once
                const cx<T> fp = pfma(fv, v, pmul(fv, vl));
                if (MODE == SEP_METRIC) {
                  if (FWD) line[r * ny + x] = mkc<T>((T)0.5 * fp.x, two ? (T)0.5 * fp.y : (T)0);
                } else {
#pragma unroll
                  for (int b = 0; b < 2; ++b) {
                    if (b && !two) break;
                    const int64_t pb = p + (int64_t)b * ny;
                    const T vb = b ? fp.y : fp.x;
                    if (MODE == SEP_GRAD || k.mode == SEP_IMAGE) {
                      ((T*)a.out)[pb] = vb;
                    } else if (k.mode == SEP_READOUT) {
                      if (ix[u][b] >= 0) ((T*)a.out)[ix[u][b]] = vb;
                    } else {  // SEP_WEIGHTS
                      const T ep = f[u][b];
                      ((T*)a.wts)[pb] = ix[u][b] < 0 ? (T)0 : (ep * ep) / vb;
                    }
                  }
                }
              }
            }
          }
        }
        __syncthreads();  // every window has been read, every image row written
      }
    } else {
      // ---- rows of the input
      for (int r = 0; r < k.rp; ++r) {
        const int row0 = 2 * (t0 + r);
        if (row0 >= nx) break;
        const bool two = row0 + 1 < nx;
        // columns loaded together: with two loads at a time the scattered readout rows of
        // 1024^2 x 1 x 3 took 52 us, now 27 (36 with two columns)
        constexpr int U = 4;
        for (int xb = tid; xb < ny; xb += U * NT) {
          T o[U][2];
          if (MODE == SEP_SKY || k.mode == SEP_COT) {
            const T* in = (const T*)a.in + (MODE == SEP_SKY
                                                ? pl * a.in_ps + (int64_t)row0 * a.in_rs
                                                : ((int64_t)pl * nx + row0) * ny);
            const int64_t rs = MODE == SEP_SKY ? a.in_rs : ny;
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
              for (int b = 0; b < 2; ++b) {
                const int x = xb + u * NT;
                o[u][b] = x < ny && (b == 0 || two) ? in[b * rs + x] : (T)0;
              }
          } else {  // SEP_COT_READOUT
            int32_t ix[U][2];
            T f[U][2];
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
              for (int b = 0; b < 2; ++b) {
                const int x = xb + u * NT;
                const int64_t p = ((int64_t)pl * nx + row0 + b) * ny + x;
                const bool ok = x < ny && (b == 0 || two);
                ix[u][b] = ok ? a.ridx[p] : -1;
                f[u][b] = ok && eps ? eps[p] : (T)1;
              }
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
              for (int b = 0; b < 2; ++b)
                o[u][b] = ix[u][b] >= 0 ? ((const T*)a.in)[ix[u][b]] : (T)0;
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
              for (int b = 0; b < 2; ++b) o[u][b] = ix[u][b] >= 0 ? f[u][b] * o[u][b] : (T)0;
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int x = xb + u * NT;
            if (x >= ny) break;
            if (MODE == SEP_SKY && a.in_exp) {
              o[u][0] = exp(o[u][0]);
              o[u][1] = two ? exp(o[u][1]) : (T)0;
            }
            line[r * ny + x] = pmul(both<T>((T)0.5), mkc<T>(o[u][0], o[u][1]));
          }
        }
      }
      __syncthreads();
    }
    // the next kernel enters beside the last item only (see sep_cols.cuh)
    if (item + (int)gridDim.x >= k.items) sep_trigger();
    if (FWD) {
      // ---- image rows -> row spectra of every window
      for (int ch = 0; ch < nchunk; ++ch) {
        const int j0 = ch * k.seqs, jn = min(k.seqs, n - j0);
        const int cnt = jn * k.rp;
#pragma unroll 1
        for (int h = 0; h < 2; h += SEQ16) {
          const int s = q0 + h + sub;
          if (sub >= SEQ16 || s >= cnt) continue;
          const int r = k.rp == 1 ? 0 : s / jn;
          const int j = j0 + s - r * jn;
          const int x0 = min(j * k.dx, k.sc_max) - k.half - k.margin + cls;
          const cx<T>* src = line + r * ny + x0;
          const bool there = 2 * (t0 + r) < nx;
          cx<T> v[16];
          if (MODE != SEP_SKY && there && x0 >= 0 && x0 + P - L1 < ny) {
#pragma unroll
            for (int q = 0; q < 16; ++q) v[q] = src[L1 * q];
          } else {
#pragma unroll
            for (int q = 0; q < 16; ++q) {
              bool in = there && (unsigned)(x0 + L1 * q) < (unsigned)ny;
              const int xa = cls + L1 * q - k.margin;
              // outside the window the value does not enter (it may be infinite)
              if (MODE == SEP_SKY) in = in && (unsigned)xa < (unsigned)k.K;
              v[q] = in ? src[L1 * q] : mkc<T>((T)0, (T)0);
              if (MODE == SEP_SKY) {
                const T w = in ? wt[xa] : (T)0;
                v[q] = mkc<T>(w * v[q].x, w * v[q].y);
              }
            }
          }
          Dft<16, false, T>::run(v);
          cx<T>* dst = buf + s * WP + 17 * cls;
#pragma unroll
          for (int q = 0; q < 16; q += 2) {
            cx<T> wa, wb;
            two_twiddles(mytw, q, wa, wb);
            dst[q] = q ? cmul<T>(v[q], wa) : v[q];
            dst[q + 1] = cmul<T>(v[q + 1], wb);
          }
        }
        __syncwarp();
        if (q0 + (lane >> 4) < cnt) row_dft_l1<T, L1, false>(buf + (q0 + (lane >> 4)) * WP, lane & 15);
        __syncwarp();
#pragma unroll 1
        for (int s = q0; s < q0 + 2 && s < cnt; ++s) {  // split the halved rows' sum
          const int r = k.rp == 1 ? 0 : s / jn, j = j0 + s - r * jn;
          const int row0 = 2 * (t0 + r);
          if (row0 >= nx) break;
          const bool two = row0 + 1 < nx;
          cx<T>* dst = (cx<T>*)a.rows + (((int64_t)pl * n + j) * nx + row0) * H + lane;
          const cx<T>* wp = buf + s * WP + slot_p;
          const cx<T>* wm = buf + s * WP + slot_m;
#pragma unroll
          for (int t = 0; t < (H + 31) / 32; ++t) {
            if (H % 32 && lane + 32 * t >= H) break;
            const bool dc = t == 0 && lane == 0;
            const cx<T> zp = wp[34 * t], zm = (dc ? wp + row_slot(H) : wm - 34 * t)[0];
            dst[32 * t] = dc ? padd(mkc<T>(zp.x, zm.x), mkc<T>(zp.x, zm.x)) : split_a<T>(zp, zm);
            if (two)
              dst[H + 32 * t] =
                  dc ? padd(mkc<T>(zp.y, zm.y), mkc<T>(zp.y, zm.y)) : split_b<T>(zp, zm);
          }
        }
        __syncwarp();  // this warp's sequences have been read
      }
      // the image rows have been read (an inverse half meets at its own barrier first)
      if (!INV) __syncthreads();
    }
  }
  if (MODE == SEP_LIKE) {
    if (a.state && a.plane0 + a.planes < a.all_planes) {  // more chunks to come
      cx<T>* st = (cx<T>*)a.state + 4 * ((int64_t)blockIdx.x * NT + tid);
      st[0] = s_lam.s;
      st[1] = s_lam.nc;
      st[2] = s_dlog.s;
      st[3] = s_dlog.nc;
      return;
    }
    __syncthreads();
    double* red = reinterpret_cast<double*>(smem_raw);  // every sequence has been read
    block_reduce2_of(s_lam.value(), s_dlog.value(), red, red + NT, a.partials, a.counter,
                     a.energy, blockIdx.x, gridDim.x);
  }
}

// bound of the numerators that the kernels divide by dx or a slab's stride
inline int64_t sep_reach(const Geom& g) { return std::max(g.nx, g.ny) + 4 * (int64_t)g.P; }

// Threads of a row CTA, and the grid: as many CTAs as fit at once, looping over the items
// (the tables are built once per CTA, and the likelihood has one partial sum per CTA).
inline int row_threads(const RowK& k) {
  return 32 * ((std::min(k.seqs, k.n * k.rp) + 1) / 2);
}
template <typename T, int L1, int MODE, bool FWD>
int row_grid(const RowK& k, size_t smem, int64_t* grid) {
  static SepKernelCache cache;
  int per_sm = 1;
  JUBIK_TRY(cache.prepare((const void*)k_sep_rows<T, L1, MODE, FWD>, row_threads(k), smem,
                          &per_sm));
  *grid = std::min<int64_t>(k.grid_items,
                            std::min<int64_t>(kSepMaxBlocks, (int64_t)sm_count() * per_sm));
  return JUBIK_OK;
}

template <typename T, int L1, int MODE, bool FWD>
int launch_rows(RowK& k, size_t smem, bool pdl, cudaStream_t s) {
  int64_t grid = 0;
  JUBIK_TRY((row_grid<T, L1, MODE, FWD>(k, smem, &grid)));
  k.base = (int)(k.item0 / grid * grid);
  return sep_launch(k_sep_rows<T, L1, MODE, FWD>, dim3((unsigned)grid), row_threads(k), smem, pdl,
                    s, "k_sep_rows", k);
}

// Kernel arguments of a launch.
template <typename T, int L1>
int row_args(const Geom& g, SepMode mode, const SepRows& a, RowK& k, size_t& smem) {
  k.a = a;
  k.mode = mode;
  k.nx = g.nx;
  k.ny = g.ny;
  k.n = g.n;
  k.dx = g.dx;
  k.half = g.half;
  k.margin = g.margin;
  k.sr_max = g.sr_max;
  k.sc_max = g.sc_max;
  k.K = g.K;
  k.scale64[0] = a.scale;
  k.scale64[1] = a.scale_lo;
  k.scale32[0] = (float)a.scale;
  k.scale32[1] = (float)(a.scale - (double)k.scale32[0] + a.scale_lo);
  const bool grad = mode == SEP_GRAD;
  k.nslab = g.n / a.slab_run;
  k.step = g.dx * a.slab_run;
  k.height = grad ? g.K : (a.slab_run - 1) * g.dx + g.P;
  // row pairs per item: as many as fill the sequences of one pass
  k.seqs = row_seqs<T, L1>(g);
  if (k.seqs < 2) {
    set_error("separable rows: %d columns exceed the shared memory", g.ny);
    return JUBIK_ERR_UNSUPPORTED;
  }
  k.rp = row_pairs(g.n, g.nx, k.seqs);
  const int pairs = (g.nx + 1) / 2;
  k.per = (pairs + k.rp - 1) / k.rp;
  if (!a.all_planes) k.a.all_planes = a.planes;  // one chunk
  const int64_t items = (int64_t)k.a.all_planes * k.per;
  if (items > 0x7fffffffLL) {
    set_error("separable rows: too many image rows for one launch");
    return JUBIK_ERR_UNSUPPORTED;
  }
  // (slabs and row spectra of a chunk are addressed by the planes of the whole image)
  const size_t row = (size_t)a.plane0 * g.n * (g.P / 2) * sizeof(cx<T>);
  if (a.slab) k.a.slab = (const char*)a.slab - row * ((size_t)k.height * k.nslab);
  if (a.rows) k.a.rows = (char*)a.rows - row * (size_t)g.nx;
  k.item0 = a.plane0 * k.per;
  k.items = (a.plane0 + a.planes) * k.per;
  k.grid_items = (int)items;
  k.late = a.slab_run == 1 ? std::max(0, (g.n - 1) * g.dx - g.sr_max) : 0;
  k.few = g.n <= k.seqs && (grad ? g.K : g.P) <= 4 * g.dx && (g.n - 1) * g.dx <= g.sc_max;
  const int64_t reach = sep_reach(g) + k.step;
  k.mul_dx = mulhi_divisor(g.dx, reach);
  k.mul_step = mulhi_divisor(k.step, reach);
  k.div_per = mulhi_divisor(k.per, items + 1);
  smem = row_smem<T, L1>(g.n, g.ny, k.rp, k.seqs);
  return JUBIK_OK;
}

template <typename T, int L1>
int dispatch_rows(const Geom& g, SepMode mode, const SepRows& a, bool pdl, cudaStream_t s) {
  RowK k{};
  size_t smem = 0;
  JUBIK_TRY((row_args<T, L1>(g, mode, a, k, smem)));
  switch (mode) {
    case SEP_SKY: return launch_rows<T, L1, SEP_SKY, true>(k, smem, pdl, s);
    case SEP_COT:
    case SEP_COT_READOUT: return launch_rows<T, L1, SEP_COT, true>(k, smem, pdl, s);
    case SEP_LIKE:
      return a.rows ? launch_rows<T, L1, SEP_LIKE, true>(k, smem, pdl, s)
                    : launch_rows<T, L1, SEP_LIKE, false>(k, smem, pdl, s);
    case SEP_METRIC: return launch_rows<T, L1, SEP_METRIC, true>(k, smem, pdl, s);
    case SEP_GRAD: return launch_rows<T, L1, SEP_GRAD, false>(k, smem, pdl, s);
    default: return launch_rows<T, L1, SEP_IMAGE, false>(k, smem, pdl, s);
  }
}

// Threads of the likelihood's launches, with or without the rows onward.
template <typename T, int L1>
int like_threads(const Geom& g, int64_t* threads) {
  SepRows a;
  a.planes = g.M * g.E;
  RowK k{};
  size_t smem = 0;
  JUBIK_TRY((row_args<T, L1>(g, SEP_LIKE, a, k, smem)));
  int64_t with = 0, without = 0;
  JUBIK_TRY((row_grid<T, L1, SEP_LIKE, true>(k, smem, &with)));
  JUBIK_TRY((row_grid<T, L1, SEP_LIKE, false>(k, smem, &without)));
  *threads = std::max(with, without) * row_threads(k);
  return JUBIK_OK;
}

}  // namespace

template <typename T>
int sep_like_threads_t(const Geom& g, int64_t* threads) {
  switch (g.P) {
    case 160: return like_threads<T, 10>(g, threads);
    case 192: return like_threads<T, 12>(g, threads);
    case 256: return like_threads<T, 16>(g, threads);
    case 320: return like_threads<T, 20>(g, threads);
    case 384: return like_threads<T, 24>(g, threads);
    case 512: return like_threads<T, 32>(g, threads);
    default: break;
  }
  set_error("separable rows do not cover P=%d", g.P);
  return JUBIK_ERR_UNSUPPORTED;
}

template <typename T>
int sep_rows_t(const Geom& g, SepMode mode, const SepRows& a, bool pdl, cudaStream_t s) {
  switch (g.P) {
    case 160: return dispatch_rows<T, 10>(g, mode, a, pdl, s);
    case 192: return dispatch_rows<T, 12>(g, mode, a, pdl, s);
    case 256: return dispatch_rows<T, 16>(g, mode, a, pdl, s);
    case 320: return dispatch_rows<T, 20>(g, mode, a, pdl, s);
    case 384: return dispatch_rows<T, 24>(g, mode, a, pdl, s);
    case 512: return dispatch_rows<T, 32>(g, mode, a, pdl, s);
    default: break;
  }
  set_error("separable rows do not cover P=%d", g.P);
  return JUBIK_ERR_UNSUPPORTED;
}

template <typename T>
bool sep_rows_fit(const Geom& g) {
  // (offsets within a patch column's slabs are 32-bit, divisions multiply-high)
  if (g.dx < 2 || sep_reach(g) * (int64_t)g.nx >= (int64_t(1) << 32) ||
      (int64_t)g.n * g.P * g.P / 2 > 0x7fffffffLL)
    return false;
  switch (g.P) {
    case 160: return row_seqs<T, 10>(g) > 0;
    case 192: return row_seqs<T, 12>(g) > 0;
    case 256: return row_seqs<T, 16>(g) > 0;
    case 320: return row_seqs<T, 20>(g) > 0;
    case 384: return row_seqs<T, 24>(g) > 0;
    case 512: return row_seqs<T, 32>(g) > 0;
    default: return false;
  }
}

}  // namespace jubik
