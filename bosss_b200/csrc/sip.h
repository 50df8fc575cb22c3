// sip.h -- face-once block kernel of scalar operators with nonlinear diffusion (sip_kernel.cuh).
#pragma once
#include "dg_kernel.cuh"
#include "dg_registry.h"

namespace bosss {

enum { VARIANT_SIP = 4 };

// launch entry for (K, Q, mode), null where there is no instance
KernelEntry sip_entry(int K, int Q, int mode);
// 1D tables of the Gauss rule with Q nodes (capi.cu)
void build_tables(int K, int Q, Tables1D& t);

}  // namespace bosss
