// Band plans of the on-chip FP32 sweep (host only).
#pragma once

#include "x2g_internal.h"

namespace x2g {

// Bands of an nni x nmu grid for clusters of `size` CTAs with `groups` threads
// per column; false where the grid is too small for them.
bool column_plan(int nni, int nmu, int size, int groups, ColPlan &plan);

}  // namespace x2g
