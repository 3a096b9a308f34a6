// Separable response: which geometries it covers, its scratch, and the dispatch
// by precision (the kernels are in sep_rows.cuh and sep_cols.cuh).
#include <algorithm>

#include "sep.h"

namespace jubik {

bool sep_supported(const Geom& g, int dtype) {
  switch (g.P) {
    case 160: case 192: case 256: case 320: case 384: case 512: break;
    default: return false;
  }
  return dtype == JUBIK_F32 ? sep_rows_fit<float>(g) : sep_rows_fit<double>(g);
}

SepSizes sep_sizes(const Geom& g, int dtype) {
  const size_t c = dtype == JUBIK_F32 ? 8 : 16, H = (size_t)g.P / 2;
  const size_t en2 = (size_t)g.E * g.n * g.n;
  SepSizes z;
  z.sky_rows = c * (size_t)g.E * g.n * g.nx * H;
  z.fwd_slabs = c * (size_t)g.M * en2 * g.P * H;  // one patch per slab; longer runs take less
  z.img_rows = c * (size_t)g.M * g.E * g.n * g.nx * H;
  z.grad_slabs = c * en2 * g.K * H;
  return z;
}

bool sep_run_fits(const Geom& g, int dtype, int run) {
  return dtype == JUBIK_F32 && (run == 2 || run == 4) && (g.P == 192 || g.P == 384) &&
         3 * g.dx == g.P && 6 * g.margin == g.P && g.nx == g.n * g.dx && g.ny == g.n * g.dx &&
         g.n % run == 0;
}

// Longer runs write fewer rows (6 strides per run of 4 patches, 12 without) and leave
// fewer to sum, but make fewer CTAs.  The longest run is taken that still leaves 1.5
// waves of CTAs, 2 with fewer than three modules, which have less to save.  A pass with
// runs of 1 / 2 / 4, in us (waves of runs of 4): 1024^2 x 7 x 3 980 / 923 / 924 (3.8),
// 1024^2 x 1 x 3 277 / 268 / 262 (3.8), 768^2 x 3 x 2 216 / 206 / 216 (1.4),
// 512^2 x 7 x 3 283 / 270 / 283 (0.95), 1024^2 x 1 x 1 117 / 113 / 115 (1.3),
// P = 384: 1024^2 x 7 x 3 1088 / 1070 / 1052 (3.8).
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
