// Linear.__call__ (nn_tfhe/Spike_LSTM.py:48-58) on either torus:
// P_A = W_j(X) A_s(X) mod X^N + 1; the LWE of coefficient 0 is a'[0] = P_A[0],
// a'[i] = -P_A[N - i] (schemas/text_jax.py:191-208), b' = P_B[0] + bias_j.
// Exact modulo 2^32 or 2^64 (words wrap around).
//
// The weight polynomials are sparse (input + hidden of N coefficients), and a
// launch has few (output, ciphertext) pairs: a block takes LIN_JT outputs of
// one ciphertext and CPT x 256 coefficients of them, compacts the coefficients
// with a nonzero weight once, and then does one shared-memory read and LIN_JT
// multiply-adds per such coefficient; A is laid out with its negated wrap in
// front, so no index is folded back in the loop.  With whole polynomials per
// block and every coefficient looked at, a tick of three requests (hidden 256,
// N = 1024) spent 0.91 ms in it, a 64-bit timestep of 16 sequences (N = 2048)
// 0.72 ms.
#pragma once

#include "tfhe_b200.h"
#include "tfhe_internal.cuh"

namespace tfhe {

constexpr int LIN_JT = 4;      // outputs per block
constexpr int LIN_NT = 256;

template <class Word>
inline size_t linear_smem(int N, int cpt) {
    return (size_t)N * (sizeof(int4) + sizeof(int)) + (size_t)(N + LIN_NT * cpt) * sizeof(Word);
}

template <class Word, class Signed, int CPT>
__global__ void __launch_bounds__(LIN_NT) linear_kernel(const int32_t* __restrict__ W, const Signed* __restrict__ bias,
                                                        int J, const Word* __restrict__ ct, int N,
                                                        Word* __restrict__ out_a, Word* __restrict__ out_b) {
    static_assert(LIN_JT == 4, "a list entry holds four weights");
    constexpr int CH = LIN_NT * CPT;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    int4* lw = reinterpret_cast<int4*>(smem_raw);               // N: weights of the listed coefficients
    int* lm = reinterpret_cast<int*>(lw + N);                   // N: the coefficients
    Word* E = reinterpret_cast<Word*>(lm + N);                  // N + CH - 1: A[c0 - (N - 1) ..], wraps negated
    __shared__ int count;
    __shared__ Word red[LIN_JT][LIN_NT / 32];
    const int tid = threadIdx.x, lane = tid & 31;
    const long long s = blockIdx.y;
    const int j0 = blockIdx.x * LIN_JT;
    const int c0 = blockIdx.z * CH;
    const Word* a_in = ct + s * 2 * N;
    const Word* b_in = a_in + N;

    if (tid == 0) count = 0;
    __syncthreads();
    // N is a multiple of 128, so every warp that enters is whole: full masks
    for (int m = tid; m < N; m += LIN_NT) {
        int w[LIN_JT];
#pragma unroll
        for (int jt = 0; jt < LIN_JT; ++jt) w[jt] = j0 + jt < J ? W[(long long)(j0 + jt) * N + m] : 0;
        const bool any = (w[0] | w[1] | w[2] | w[3]) != 0;
        const unsigned vote = __ballot_sync(0xffffffffu, any);
        int at = 0;
        if (lane == 0 && vote) at = atomicAdd(&count, __popc(vote));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(vote & ((1u << lane) - 1u));
        if (any) {
            lm[at] = m;
            lw[at] = make_int4(w[0], w[1], w[2], w[3]);
        }
    }
    for (int i = tid; i < N + CH - 1; i += LIN_NT) {
        const int c = c0 - (N - 1) + i;
        if (c < N) E[i] = c >= 0 ? a_in[c] : (Word)0 - a_in[c + N];
    }
    __syncthreads();
    const int n = count;

    Word acc[LIN_JT][CPT];
#pragma unroll
    for (int jt = 0; jt < LIN_JT; ++jt)
#pragma unroll
        for (int r = 0; r < CPT; ++r) acc[jt][r] = 0;
    const Word* e0 = E + (N - 1) + tid;
#pragma unroll 4
    for (int i = 0; i < n; ++i) {
        const int4 w = lw[i];
        const Word* e = e0 - lm[i];
#pragma unroll
        for (int r = 0; r < CPT; ++r) {
            const Word v = e[LIN_NT * r];
            acc[0][r] += (Word)(Signed)w.x * v;
            acc[1][r] += (Word)(Signed)w.y * v;
            acc[2][r] += (Word)(Signed)w.z * v;
            acc[3][r] += (Word)(Signed)w.w * v;
        }
    }
#pragma unroll
    for (int jt = 0; jt < LIN_JT; ++jt) {
        const int j = j0 + jt;
        if (j >= J) break;
        Word* dst = out_a + (s * J + j) * (long long)N;
#pragma unroll
        for (int r = 0; r < CPT; ++r) {
            const int c = c0 + tid + LIN_NT * r;
            if (c == 0) dst[0] = acc[jt][r];
            else if (c < N) dst[N - c] = (Word)0 - acc[jt][r];
        }
    }

    // b' = sum_m W[m] B[-m]: B[0] for m = 0, -B[N - m] otherwise
    if (blockIdx.z != 0) return;
    Word pb[LIN_JT] = {0, 0, 0, 0};
    for (int i = tid; i < n; i += LIN_NT) {
        const int m = lm[i];
        const Word bv = m == 0 ? b_in[0] : (Word)0 - b_in[N - m];
        const int4 w = lw[i];
        pb[0] += (Word)(Signed)w.x * bv;
        pb[1] += (Word)(Signed)w.y * bv;
        pb[2] += (Word)(Signed)w.z * bv;
        pb[3] += (Word)(Signed)w.w * bv;
    }
#pragma unroll
    for (int jt = 0; jt < LIN_JT; ++jt) {
        Word v = pb[jt];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) red[jt][tid >> 5] = v;
    }
    __syncthreads();
    if (tid < LIN_JT && j0 + tid < J) {
        Word v = (Word)bias[j0 + tid];
        for (int w = 0; w < LIN_NT / 32; ++w) v += red[tid][w];
        out_b[s * J + j0 + tid] = v;
    }
}

// coefficients per thread: as many as leave about two blocks per SM and do not
// reach past N (N = 128, 1000 outputs of 40 ciphertexts, dense, 64 bits: 450 us, 1622
// with four)
template <class Word, class Signed>
int launch_linear(const int32_t* W, const Signed* bias, int J, const Word* ct, long long S, int N, Word* out_a,
                  Word* out_b, cudaStream_t stream) {
    const long long tiles = (long long)((J + LIN_JT - 1) / LIN_JT) * S;
    int cpt = 4;
    while (cpt > 1 && LIN_NT * cpt > N) cpt /= 2;
    while (cpt > 1 && tiles * ((N + LIN_NT * cpt - 1) / (LIN_NT * cpt)) < 2 * sm_count()) cpt /= 2;
    auto kern = cpt == 4 ? linear_kernel<Word, Signed, 4> : cpt == 2 ? linear_kernel<Word, Signed, 2>
                                                                     : linear_kernel<Word, Signed, 1>;
    const size_t smem = linear_smem<Word>(N, cpt);
    TFHE_TRY(smem_attr_once((const void*)kern, smem));
    const dim3 grid((J + LIN_JT - 1) / LIN_JT, (unsigned)S, (N + LIN_NT * cpt - 1) / (LIN_NT * cpt));
    count_launch();
    kern<<<grid, LIN_NT, smem, stream>>>(W, bias, J, ct, N, out_a, out_b);
    return check_cuda(cudaGetLastError(), "linear kernel launch");
}

}  // namespace tfhe
