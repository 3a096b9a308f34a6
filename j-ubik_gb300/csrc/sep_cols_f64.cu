// Separable column kernels in FP64.
#include "sep_cols.cuh"

namespace jubik {
template int sep_cols_t<double>(const Geom&, SepColsKind, const SepCols&, bool, cudaStream_t);
}  // namespace jubik
