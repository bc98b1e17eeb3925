#include "x2g_columns.cuh"

namespace x2g {

// Up to 11 warps per group, two groups of threads per CTA.
ColKernel column_kernel_split(int slots, bool sep) {
  if (sep && slots <= 2) return {(const void *)k_columns<2, true, 352, 2, 1>, 2};
  if (!sep && slots <= 2) return {(const void *)k_columns<2, false, 352, 2, 1>, 2};
  if (sep && slots <= 3) return {(const void *)k_columns<3, true, 352, 2, 1>, 3};
  if (!sep && slots <= 3) return {(const void *)k_columns<3, false, 352, 2, 1>, 3};
  if (sep && slots <= 4) return {(const void *)k_columns<4, true, 352, 2, 1>, 4};
  if (!sep && slots <= 4) return {(const void *)k_columns<4, false, 352, 2, 1>, 4};
  if (sep && slots <= 5) return {(const void *)k_columns<5, true, 352, 2, 1>, 5};
  if (!sep && slots <= 5) return {(const void *)k_columns<5, false, 352, 2, 1>, 5};
  if (sep && slots <= 6) return {(const void *)k_columns<6, true, 352, 2, 1>, 6};
  if (!sep && slots <= 6) return {(const void *)k_columns<6, false, 352, 2, 1>, 6};
  return {nullptr, slots};
}

}  // namespace x2g
