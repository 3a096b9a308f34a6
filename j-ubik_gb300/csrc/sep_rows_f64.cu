// Separable row kernels in FP64.
#include <algorithm>

#include "sep_rows.cuh"

namespace jubik {
template int sep_rows_t<double>(const Geom&, SepMode, const SepRows&, bool, cudaStream_t);
template bool sep_rows_fit<double>(const Geom&);
template int sep_like_threads_t<double>(const Geom&, int64_t*);
}  // namespace jubik
