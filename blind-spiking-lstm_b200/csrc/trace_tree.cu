// Instantiations and launches of the trace at N = 2048 on the 64-bit torus.
#include "trace_tree.cuh"

#include <cstdlib>

#include "tfhe_b200.h"
#include "tfhe_dispatch.h"

namespace tfhe {

// Levels 4 to 6: the digit bits and two more in a float64's 53, and products
// of the 22-bit limbs below 2^43.  TFHE_B200_TRACE_TREE=0 keeps new keys with
// the general kernel.
bool trace_tree_takes(int N, int l, int log2_beta) {
    const char* env = getenv("TFHE_B200_TRACE_TREE");
    if (env && env[0] == '0') return false;
    return N == TT_N && l >= 4 && l <= 6 && l * log2_beta <= 50 &&
           (long long)N * l * (1LL << (log2_beta - 1)) * (1LL << 21) <= (1LL << 43);
}

size_t trace_tree_key_words(int l, int steps) { return (size_t)steps * TT_NO * l * TT_H; }

int trace_tree_key(const unsigned long long* keys, int l, int steps, const FftPlan* pl, double2* dst, cudaStream_t stream) {
    count_launch();
    trace_key_kernel<<<dim3((unsigned)(steps * l * 2), TT_LIMBS), 256, TT_H * sizeof(double2), stream>>>(
        keys, l, pl->qt, pl->tw, pl->freq, dst);
    return check_cuda(cudaGetLastError(), "galois key layout launch");
}

int launch_trace_tree(const unsigned long long* lwe_a, const unsigned long long* lwe_b, const double2* key, int l, int log2_beta, int steps, long long R,
                      unsigned long long* out, const FftPlan* pl, cudaStream_t stream) {
    auto kern = l == 4 ? trace_tree_kernel<4> : l == 5 ? trace_tree_kernel<5> : trace_tree_kernel<6>;
    TFHE_TRY(smem_attr_once((const void*)kern, trace_tree_smem(l)));
    const TraceTreeArgs a{lwe_a, lwe_b, key, pl->qt, pl->tw, log2_beta, steps, R, out};
    count_launch();
    kern<<<(unsigned)R, TT_THREADS, trace_tree_smem(l), stream>>>(a);
    return check_cuda(cudaGetLastError(), "trace launch");
}

}  // namespace tfhe
