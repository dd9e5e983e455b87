// Instantiations of the shared-key cluster kernel at N = 2048 (br_share.cuh).
#include "br_share.cuh"
#include "tfhe_dispatch.h"

namespace tfhe {

BrKernel br_share_kernel_for(bool t64) { return t64 ? br_share_kernel<true> : br_share_kernel<false>; }
BrKernel br_share_lost() { return br_share_kernel<false, true>; }

}  // namespace tfhe
