// Separable column kernels in FP32.
#include "sep_cols.cuh"

namespace jubik {
template int sep_cols_t<float>(const Geom&, SepColsKind, const SepCols&, bool, cudaStream_t);
double sep_run_waves(const Geom& g, int run) {
  return g.P == 192 ? run_waves<float, 12>(g, run) : run_waves<float, 24>(g, run);
}
}  // namespace jubik
