// The complex128 reverse turning-pass kernels (csrc/bk_adj_turn.cuh).
#include "bk_adj_turn.cuh"

namespace bk {
const void* adj_turn_kernel_f64(int tb, int w2, int w3) { return adj_turn_table<double>(tb, w2, w3); }
}  // namespace bk
