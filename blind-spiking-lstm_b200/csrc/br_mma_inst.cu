// Instantiations of the matrix-instruction blind rotations at N = 1024.
// Compiled twice, for the native buffers (BM_REF = 0) and for the drop-in's
// (BM_REF = 1), so that the two build in parallel.
#include "br_mma_cluster.cuh"
#include "tfhe_dispatch.h"

#ifndef BM_REF
#error "BM_REF must be defined (0: native buffers, 1: the drop-in's)"
#endif

namespace tfhe {

template <int L, int T>
static BrKernel of(int C) {
    switch (C) {
        case 1: return br_mma_kernel<L, T, BM_REF != 0>;
        case 2: return br_mma_cluster_kernel<L, T, 2, BM_REF != 0>;
        case 4: return br_mma_cluster_kernel<L, T, 4, BM_REF != 0>;
        case 8: return br_mma_cluster_kernel<L, T, 8, BM_REF != 0>;
        default: return nullptr;
    }
}

static BrKernel pick(int L, int M, int C) {
    if (M != 4 && M != 8) return nullptr;
    if (L == 2) return M == 8 ? of<2, 2>(C) : of<2, 1>(C);
    if (L == 3) return M == 8 ? of<3, 2>(C) : of<3, 1>(C);
    return nullptr;
}

#if BM_REF
BrKernel br_mma_ref(int L, int M, int C) { return pick(L, M, C); }
BmRefConvKernel bm_ref_key() { return bm_ref_key_kernel; }
#else
BrKernel br_mma_native(int L, int M, int C) { return pick(L, M, C); }
BrKernel br_mma_lost() { return br_mma_cluster_kernel<3, 2, 8, false, true>; }
BmConvKernel bm_key() { return bm_key_kernel; }

size_t br_mma_smem_for(int L, int M, int C) {
    switch (C) {
        case 1: return br_mma_smem(L, M);
        case 2: return L == 2 ? br_mma_cluster_smem<2, 2>(M) : br_mma_cluster_smem<3, 2>(M);
        case 4: return L == 2 ? br_mma_cluster_smem<2, 4>(M) : br_mma_cluster_smem<3, 4>(M);
        default: return L == 2 ? br_mma_cluster_smem<2, 8>(M) : br_mma_cluster_smem<3, 8>(M);
    }
}
#endif

}  // namespace tfhe
