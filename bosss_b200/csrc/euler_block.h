// euler_block.h -- face-once block kernel of the 3D Euler operator (euler_block.cuh).
#pragma once
#include "dg_kernel.cuh"
#include "dg_registry.h"

namespace bosss {

enum { VARIANT_EULER_BLOCK = 5 };

// launch entry for (K, Q, mode); null where there is no instance (Q != K + 1)
KernelEntry euler_block_entry(int K, int Q, int mode);

}  // namespace bosss
