// Separable row kernels in FP32.
#include <algorithm>

#include "sep_rows.cuh"

namespace jubik {
template int sep_rows_t<float>(const Geom&, SepMode, const SepRows&, bool, cudaStream_t);
template bool sep_rows_fit<float>(const Geom&);
template int sep_like_threads_t<float>(const Geom&, int64_t*);
}  // namespace jubik
