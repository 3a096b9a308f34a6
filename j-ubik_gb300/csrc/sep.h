// Separable evaluation of the patch response: declarations shared by the row
// kernels (sep_rows.cuh), the column kernels (sep_cols.cuh) and the C ABI.
//
// The response of a patch is a 2-D circular convolution of side P, and the
// patches overlap-add (jubik/convolve.py:86-145).  Both steps are linear and
// act on rows and columns separately, so
//   forward:  R = rowsum_j  F_x^-1  colsum_i  F_y^-1  H  F_y  w_y  F_x  w_x
//   adjoint:  the transpose, factor by factor,
// where i and j run over the patch rows and columns.  The sum over vertically
// overlapping patches (i) commutes with the row transform F_x, and the patches
// of one patch column j cut the same image rows.  Every image row is therefore
// transformed once per patch column, not once per patch that covers it: P / dx
// (3 at P = 3 dx) times fewer row transforms, and what crosses between patches
// is summed in a fixed order in registers and shared memory.  Columns are
// independent of one another through the PSF product and the module sum, so
// a CTA of the column kernels holds P rows of a few columns only, and several
// CTAs share an SM whatever P is.
//
// Between the two kinds of kernels travel row spectra: per image row and patch
// column the P / 2 complex values kx = 0 .. P/2 - 1 of the row's window, the
// kx = 0 and kx = P/2 values (real for a real row) packed into column 0.
#pragma once

#include <vector>

#include "internal.h"

namespace jubik {

// What a row kernel does with the image rows it sums up or starts from.
enum SepMode {
  SEP_SKY = 0,      // start: sky rows (or exp of log-sky rows), weighted by the window
  SEP_COT,          // start: an (M, E, nx, ny) cotangent image
  SEP_COT_READOUT,  // start: a readout vector, scattered and multiplied by the exposure
  SEP_IMAGE,        // end: the image
  SEP_READOUT,      // end: exposure times the image, gathered into readout order
  SEP_LIKE,         // likelihood terms, metric weights and, onwards, the residual rows
  SEP_METRIC,       // onwards: the metric weights times the image
  SEP_WEIGHTS,      // end: metric weights of lam = exposure times the image
  SEP_GRAD          // end: window-weighted sum of the patches, the sky gradient
};

struct SepRows {
  const void* in = nullptr;    // SEP_SKY / SEP_COT / SEP_COT_READOUT input
  int64_t in_rs = 0, in_ps = 0;  // SEP_SKY: row and plane strides
  int in_exp = 0;              // SEP_SKY: the sky is exp of the input
  const void* slab = nullptr;  // column-summed spectra of the patches (or runs of patches)
  int slab_run = 1;            // patches per slab
  void* rows = nullptr;        // row spectra written (planes, n, nx, P / 2), or nullptr
  void* out = nullptr;         // SEP_IMAGE / SEP_READOUT / SEP_GRAD output
  const void* tw = nullptr;    // (P) twiddles
  const void* wt = nullptr;    // (K) window weights
  const void* eps = nullptr;
  const int32_t* dimg = nullptr;
  const int32_t* ridx = nullptr;
  void* wts = nullptr;
  double* partials = nullptr;
  unsigned int* counter = nullptr;
  double* energy = nullptr;
  double scale = 1.0, scale_lo = 0.0;  // the factor's two words
  // Planes of the images (M E, or E for SEP_SKY and SEP_GRAD), and the module chunk of them
  // that this launch takes: `planes` from plane0.  Slabs and row spectra hold the chunk only.
  int all_planes = 0, plane0 = 0, planes = 0;
  // SEP_LIKE in several chunks: per thread the sums of the chunks before (sep_state_bytes).
  // Every launch has the grid of the whole image, and a CTA the items that it would take
  // there, so the energy has the same bits however the modules are cut.
  void* state = nullptr;
};

// Adjoint columns of a module chunk: the sums of the chunks before are read (RESUME), and
// passed on instead of going to the gradient slabs (PASS_ON).  They lie behind the slabs.
enum { SEP_RESUME = 1 << 8, SEP_PASS_ON = 1 << 9 };
struct SepCols {
  const void* rows = nullptr;  // row spectra read
  const void* hmain = nullptr;
  const void* hnyq = nullptr;
  const void* tw = nullptr;
  const void* wt = nullptr;
  void* slab = nullptr;        // slabs written
  // forward: patches per slab; adjoint of a module chunk: SEP_RESUME | SEP_PASS_ON.  (More
  // arguments, even unused ones, made the adjoint spill: 249 -> 261 us at 1024^2 x 7 x 3.)
  int run = 1;
};

// FFT sides the separable kernels cover, given their shared memory for this
// field (rows of ny pixels).
bool sep_supported(const Geom& g, int dtype);
// Scratch of a plan, in bytes: sky row spectra, forward slabs of `run` patches, image row
// spectra, gradient slabs; module sums between chunks.
struct SepSizes {
  size_t sky_rows, fwd_slabs, img_rows, grad_slabs;
  size_t acc;  // several chunks only
};
// (of `modules` modules at once)
SepSizes sep_sizes(const Geom& g, int dtype, int run, int modules);
// Bytes of the likelihood's sums between chunks: four complex values a thread.
int sep_state_bytes(const Geom& g, int dtype, size_t* bytes);
// Gains less one of the column transforms (gy, by ky) and of the row transforms (gx, by kx)
// of side P, each forward and back: P values each.
void sep_gains(int P, std::vector<double>& gy, std::vector<double>& gx);
// Blocks of the likelihood's row kernel at most (its partial sums).
constexpr int kSepMaxBlocks = 2048;

int sep_rows(const Geom& g, int dtype, SepMode mode, const SepRows& a, bool pdl, cudaStream_t s);
// SEP_COLS_FWD: sky row spectra -> slabs of a.run patches each;
// SEP_COLS_ADJ: image row spectra -> module sum -> gradient slabs
enum SepColsKind { SEP_COLS_FWD, SEP_COLS_ADJ };
int sep_cols(const Geom& g, int dtype, SepColsKind kind, const SepCols& a, bool pdl,
             cudaStream_t s);

// per-precision parts (one translation unit each)
template <typename T>
int sep_rows_t(const Geom& g, SepMode mode, const SepRows& a, bool pdl, cudaStream_t s);
template <typename T>
bool sep_rows_fit(const Geom& g);
template <typename T>
int sep_like_threads_t(const Geom& g, int64_t* threads);
template <typename T>
int sep_cols_t(const Geom& g, SepColsKind kind, const SepCols& a, bool pdl, cudaStream_t s);

// Whether forward slabs of `run` (2 or 4) patches exist: FP32, P = 192 or 384 from strides
// of P / 3 rows and margins of P / 6, a field of whole strides, runs that tile the columns.
bool sep_run_fits(const Geom& g, int dtype, int run);
// The run length the library takes.
int sep_auto_run(const Geom& g, int dtype);
double sep_run_waves(const Geom& g, int run);  // waves of CTAs (sep_run_fits geometries)

}  // namespace jubik
