// Separable response: which geometries it covers, its scratch, and the dispatch
// by precision (the kernels are in sep_rows.cuh and sep_cols.cuh).
#include <algorithm>
#include <cmath>
#include <complex>
#include <vector>

#include "sep.h"

namespace jubik {

bool sep_supported(const Geom& g, int dtype) {
  switch (g.P) {
    case 160: case 192: case 256: case 320: case 384: case 512: break;
    default: return false;
  }
  return dtype == JUBIK_F32 ? sep_rows_fit<float>(g) : sep_rows_fit<double>(g);
}

SepSizes sep_sizes(const Geom& g, int dtype, int run, int modules) {
  const size_t c = dtype == JUBIK_F32 ? 8 : 16, H = (size_t)g.P / 2;
  const size_t en2 = (size_t)g.E * g.n * g.n;
  SepSizes z;
  z.sky_rows = c * (size_t)g.E * g.n * g.nx * H;
  z.fwd_slabs = c * (size_t)modules * g.E * g.n * (g.n / run) * ((run - 1) * g.dx + g.P) * H;
  z.img_rows = c * (size_t)modules * g.E * g.n * g.nx * H;
  z.grad_slabs = c * en2 * g.K * H;
  z.acc = c * en2 * g.P * H;
  return z;
}

int sep_state_bytes(const Geom& g, int dtype, size_t* bytes) {
  int64_t threads = 0;
  JUBIK_TRY(dtype == JUBIK_F32 ? sep_like_threads_t<float>(g, &threads)
                               : sep_like_threads_t<double>(g, &threads));
  *bytes = (size_t)threads * 4 * (dtype == JUBIK_F32 ? 8 : 16);
  return JUBIK_OK;
}

// The transforms' constants are rounded to FP32, so a transform and its inverse return
// (1 + g) of a frequency, not all of it.  At side 192 g is -0.59e-7 in the mean along rows
// and as much along columns, alike for nearly every frequency but the constant one: of the
// back-projection's error against 64 bits (1.84e-7) 1.09e-7 was this one factor.  The PSF
// spectra, which are computed in FP64, take the factor back before they are rounded
// (errors before -> now at 1024^2: gradient 7.3e-7 -> 3.8e-7, metric product 3.5e-7 ->
// 1.8e-7, back-projection 1.68e-7 -> 1.46e-7).
// Each transform of side 16 L1 multiplies an element by one entry of the 16-point matrix,
// one twiddle and one entry of the L1-point matrix, and its inverse by their conjugates:
// the gain is the mean of the three squared magnitudes over the elements.
namespace {
using Cx = std::complex<double>;
Cx rounded_root(int k, int N) {  // exp(-2 pi i k / N) with its parts rounded to FP32
  const double a = -2.0 * 3.14159265358979323846 * (double)(k % N) / N;
  return Cx((float)std::cos(a), (float)std::sin(a));
}
// the matrix of the N-point codelet (fft_codelets.cuh), row by row
std::vector<Cx> codelet_matrix(int N) {
  std::vector<Cx> m((size_t)N * N);
  int n1 = 0;
  switch (N) {
    case 8: case 16: case 20: case 32: n1 = 4; break;
    case 12: case 24: n1 = 3; break;
    case 10: n1 = 5; break;
    default: break;  // no factors
  }
  if (!n1) {
    for (int k = 0; k < N; ++k)
      for (int n = 0; n < N; ++n) m[k * N + n] = rounded_root(k * n, N);
    return m;
  }
  const int n2 = N / n1;
  const std::vector<Cx> a = codelet_matrix(n1), b = codelet_matrix(n2);
  for (int i = 0; i < n2; ++i)
    for (int k1 = 0; k1 < n1; ++k1)
      for (int n = 0; n < n1; ++n)
        for (int k2 = 0; k2 < n2; ++k2)
          m[(size_t)(k1 + n1 * k2) * N + n2 * n + i] =
              a[k1 * n1 + n] * rounded_root(i * k1, N) * b[k2 * n2 + i];
  return m;
}
// squared magnitudes less one
double excess(Cx z) { return std::norm(z) - 1.0; }
}  // namespace

void sep_gains(int P, std::vector<double>& gy, std::vector<double>& gx) {
  const int L1 = P / 16;
  const std::vector<Cx> a = codelet_matrix(16), b = codelet_matrix(L1);
  std::vector<double> ea(16, 0.0), eb(L1, 0.0);  // means over a matrix row
  for (int k = 0; k < 16; ++k)
    for (int n = 0; n < 16; ++n) ea[k] += excess(a[k * 16 + n]) / 16;
  for (int k = 0; k < L1; ++k)
    for (int n = 0; n < L1; ++n) eb[k] += excess(b[k * L1 + n]) / L1;
  // (first order: the excesses add)
  std::vector<double> g(P);
  gy.assign(P, 0.0);
  gx.assign(P, 0.0);
  for (int c = 0; c < L1; ++c)
    for (int q = 0; q < 16; ++q) {
      double over_n = 0.0, over_c = 0.0;
      for (int i = 0; i < 16; ++i) over_n += excess(rounded_root(c * i, P)) / 16;
      for (int i = 0; i < L1; ++i) over_c += excess(rounded_root(i * q, P)) / L1;
      gy[c + L1 * q] = eb[c] + over_n + ea[q];   // columns: class c, then slot q
      g[q + 16 * c] = ea[q] + over_c + eb[c];    // rows: slot q, then class c
    }
  // two real rows travel as one sequence: kx and P - kx serve both
  for (int k = 0; k < P; ++k) gx[k] = 0.5 * (g[k] + g[(P - k) % P]);
}

bool sep_run_fits(const Geom& g, int dtype, int run) {
  return dtype == JUBIK_F32 && (run == 2 || run == 4) && (g.P == 192 || g.P == 384) &&
         3 * g.dx == g.P && 6 * g.margin == g.P && g.nx == g.n * g.dx && g.ny == g.n * g.dx &&
         g.n % run == 0;
}

// Longer runs write fewer rows (6 strides per run of 4 patches, 12 without) and leave
// fewer to sum, but make fewer CTAs.  The longest run is taken that still leaves 1.5
// waves of CTAs, 2 with fewer than three modules.  A pass with runs of 1 / 2 / 4, in us
// (waves of runs of 4): 1024^2 x 7 x 3 909 / 869 / 855 (3.8), 768^2 x 3 x 2 190 / 183 / 191
// (1.4), 512^2 x 7 x 3 260 / 254 / 265 (0.95); of 1 and of the run taken: 1024^2 x 1 x 3
// 241 / 225 (4; 3.8), 1024^2 x 1 x 1 97 / 95 (2; 1.3), P = 384 1024^2 x 7 x 3 970 / 875
// (4; 3.8).  Few modules gain little: at 512^2 x 2 x 3 (1.9 waves of runs of 2) all lie
// within 1.3 %, 104.3 / 103.7 / 105.1, so the line between 1 and 2 could lie on either side.
int sep_auto_run(const Geom& g, int dtype) {
  const double least = g.M >= 3 ? 1.5 : 2.0;
  for (const int r : {4, 2})
    if (sep_run_fits(g, dtype, r) && sep_run_waves(g, r) >= least) return r;
  return 1;
}

int sep_rows(const Geom& g, int dtype, SepMode mode, const SepRows& a, bool pdl, cudaStream_t s) {
  return dtype == JUBIK_F32 ? sep_rows_t<float>(g, mode, a, pdl, s)
                            : sep_rows_t<double>(g, mode, a, pdl, s);
}

int sep_cols(const Geom& g, int dtype, SepColsKind kind, const SepCols& a, bool pdl,
             cudaStream_t s) {
  return dtype == JUBIK_F32 ? sep_cols_t<float>(g, kind, a, pdl, s)
                            : sep_cols_t<double>(g, kind, a, pdl, s);
}

}  // namespace jubik
