// Separable column kernels in FP32.
#include "sep_cols.cuh"

namespace jubik {
template int sep_cols_t<float>(const Geom&, SepColsKind, const SepCols&, bool, cudaStream_t);
}  // namespace jubik
