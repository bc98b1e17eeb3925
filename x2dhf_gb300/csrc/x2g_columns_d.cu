#include "x2g_columns.cuh"

namespace x2g {

// Up to 17 warps.
ColKernel column_kernel_broad(int slots, bool sep) {
  if (sep && slots <= 5) return {(const void *)k_columns<5, true, 544, 1, 1>, 5};
  if (!sep && slots <= 5) return {(const void *)k_columns<5, false, 544, 1, 1>, 5};
  if (sep && slots <= 7) return {(const void *)k_columns<7, true, 544, 1, 1>, 7};
  if (!sep && slots <= 7) return {(const void *)k_columns<7, false, 544, 1, 1>, 7};
  if (sep && slots <= 10) return {(const void *)k_columns<10, true, 544, 1, 1>, 10};
  if (!sep && slots <= 8) return {(const void *)k_columns<8, false, 544, 1, 1>, 8};
  return {nullptr, slots};
}

}  // namespace x2g
