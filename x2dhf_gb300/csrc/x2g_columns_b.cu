#include "x2g_columns.cuh"

namespace x2g {

// Potentials, two CTAs per SM, up to 11 warps.
ColKernel column_kernel_pair(int slots, bool sep) {
  if (sep && slots <= 5) return {(const void *)k_columns<5, true, 352, 1, 2>, 5};
  if (sep && slots <= 7) return {(const void *)k_columns<7, true, 352, 1, 2>, 7};
  if (sep && slots <= 9) return {(const void *)k_columns<9, true, 352, 1, 2>, 9};
  return {nullptr, slots};
}

}  // namespace x2g
