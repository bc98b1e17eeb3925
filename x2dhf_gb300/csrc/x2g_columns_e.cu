#include "x2g_columns.cuh"

namespace x2g {

// Up to 8 warps per group, two groups of threads per CTA.
ColKernel column_kernel_slim(int slots, bool sep) {
  if (sep && slots <= 6) return {(const void *)k_columns<6, true, 256, 2, 1>, 6};
  if (!sep && slots <= 6) return {(const void *)k_columns<6, false, 256, 2, 1>, 6};
  if (sep && slots <= 8) return {(const void *)k_columns<8, true, 256, 2, 1>, 8};
  if (!sep && slots <= 8) return {(const void *)k_columns<8, false, 256, 2, 1>, 8};
  if (sep && slots <= 10) return {(const void *)k_columns<10, true, 256, 2, 1>, 10};
  if (!sep && slots <= 10) return {(const void *)k_columns<10, false, 256, 2, 1>, 10};
  return {nullptr, slots};
}

}  // namespace x2g
