#include "x2g_columns.cuh"

namespace x2g {

// Up to 5 warps per group, two groups of threads per CTA.
ColKernel column_kernel_thin(int slots, bool sep) {
  if (sep && slots <= 12) return {(const void *)k_columns<12, true, 160, 2, 1>, 12};
  if (!sep && slots <= 12) return {(const void *)k_columns<12, false, 160, 2, 1>, 12};
  if (sep && slots <= 16) return {(const void *)k_columns<16, true, 160, 2, 1>, 16};
  if (!sep && slots <= 16) return {(const void *)k_columns<16, false, 160, 2, 1>, 16};
  return {nullptr, slots};
}

// Up to 25 warps.
ColKernel column_kernel_flat(int slots, bool sep) {
  if (sep && slots <= 4) return {(const void *)k_columns<4, true, 800, 1, 1>, 4};
  if (!sep && slots <= 4) return {(const void *)k_columns<4, false, 800, 1, 1>, 4};
  return {nullptr, slots};
}

}  // namespace x2g
