// The complex128 turning-pass kernels (csrc/bk_alt.cuh), one source per precision so that they build in parallel.
#include "bk_alt.cuh"

namespace bk {
const void* alt_kernel_f64(int tb, int w2, int w3, bool batch) { return alt_kernel_table<double>(tb, w2, w3, batch); }
}  // namespace bk
