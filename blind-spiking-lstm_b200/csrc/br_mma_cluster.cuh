// The matrix-instruction blind rotation (br_mma.cuh) for batches under a
// round: four ciphertexts per cluster of C CTAs (C = 2, 4, 8).
//
// A CTA's time per group in br_mma_kernel is that of the transforms of its
// four ciphertexts and of the contraction of all points; with fewer
// ciphertexts than four per SM the SMs idle or the columns do.  Here CTA r of
// a cluster transforms its share of the four ciphertexts (C = 2: two; C = 4:
// one; C = 8: one polynomial of one) and contracts 1/C of the points for all
// four, so each SM reads 1/C of a group's key and the columns stay full:
//   * the forward inner pass sends its blocks to the points' owners and the
//     contraction its results to the CTA that holds the ciphertext's polynomial
//     (distributed shared memory, stores only, so no remote read waits on the
//     way; 512 bytes in a row per store: 16-byte pieces of scattered rows took
//     a third longer);
//   * C >= 4: st.async stores counted on an mbarrier of the receiving CTA, one
//     for the digits of its points, one for its outputs, each waited for once
//     per group (a cluster barrier's release waits for a fence of more than a
//     thousand cycles); the results are gathered in the CTA first.  C = 2, whose
//     shared memory is full: plain stores and two cluster barriers a group.
// The key words of a warp's first points of the next group are copied to shared
// memory (cp.async, each lane its own words) while that group's transform
// runs: registers held for them that long would be spilled, and waited for.
// For C >= 4 the L digit levels of a polynomial go to L groups of 64 threads,
// each holding the accumulator (computed L times over) and taking its level.
//
// Shared memory is single-buffered.  C = 2: digits of group g + 1 reach an owner
// only after the second barrier of group g, which follows its reads of group
// g; outputs of group g + 1 reach a polynomial's CTA after the first barrier of
// g + 1, which follows its reads of group g.  C >= 4: a CTA sends digits of group
// g + 1 only when all its outputs of group g have come, to which every warp of
// every CTA contributes after its reads of the digits of group g; and it is
// sent outputs of g + 1 only by CTAs that hold all digits of g + 1, among them
// its own, which it sends after its reads of the outputs of group g.  A barrier
// of the CTA lies between two waits for the same mbarrier, and the second phase
// needs this CTA's own stores, so no thread misses a phase.
//
// n=630 N=1024 with the key switch, ms: batch 1 1.11 (one ciphertext on eight
// CTAs, br_cluster_kernel, 1.58), 32 1.12 (on four CTAs 1.61), 60 1.15 (cluster
// pair 1.93), 128 1.97 (one CTA each 2.50), 256 2.89 (two per CTA 4.20); the
// launcher leaves 61 to 74 to the pair (1.83) and 133 to 148 to one CTA each (2.40).
// A group at C = 8 takes 10.3k cycles: about 3.5k the contraction (1.5k of it
// matrix issue), the rest the chain of passes and exchanges (FP64 pipe 19%, FP64
// matrix pipe 15%).
#pragma once

#include "br_mma.cuh"
#include "br_split.cuh"

namespace tfhe {

template <int L, int C>
struct BmcShape {
    static constexpr int P = 2 * L;
    static constexpr int NC = C == 2 ? 2 : 1;                        // ciphertexts per CTA
    static constexpr int NA = 8 / C;                                 // accumulator polynomials per CTA
    static constexpr int ND = NA * L;                                // digit polynomials per CTA
    static constexpr int PPC = BM_H / C;                             // points per CTA
    static constexpr bool LP = C >= 4;                               // levels side by side
    // C = 2: outputs in place of their level-0 digits (same points, same thread)
    static constexpr int OUT = C == 2 ? 0 : NA;
    // pairs of a warp's points whose key words are copied to shared memory
    // during the transform: as many as fit beside the spectra
    static constexpr int STAGED = C == 8 ? 2 : (C == 4 ? 1 : 0);
    // exchange by counted stores (C >= 4), results gathered in the CTA first
    static constexpr bool ASYNC = C >= 4;
    static constexpr int GATHER = ASYNC ? 8 * PPC : 0;
};

template <int L, int C>
inline size_t br_mma_cluster_smem(int M) {
    using S = BmcShape<L, C>;
    return (size_t)((S::ND + S::OUT) * BM_H + BM_K * S::P * S::PPC + 16 * S::STAGED * (M / 4) * L * 32 + S::GATHER) *
               sizeof(double2) +
           (size_t)(BM_N + Plan<9>::TW + (8 + 64) * BM_NODE) * sizeof(double2) +
           (size_t)BM_ROT_GROUPS * M * BM_K * sizeof(uint16_t) + 2 * sizeof(uint64_t) + 2 * sizeof(int) + 16;
}

__device__ __forceinline__ void st_peer(uint32_t addr, double2 v) {
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(addr), "d"(v.x), "d"(v.y) : "memory");
}

__device__ __forceinline__ void st_peer(uint32_t addr, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}

// store into another CTA's shared memory, its bytes counted on that CTA's
// mbarrier as they land (no fence: barrier.cluster's release costs more than a
// thousand cycles here)
__device__ __forceinline__ void st_async(uint32_t addr, double2 v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(addr),
                 "d"(v.x), "d"(v.y), "r"(bar)
                 : "memory");
}

__device__ __forceinline__ void st_async(uint32_t addr, double v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(addr), "d"(v),
                 "r"(bar)
                 : "memory");
}

// wait for phase `parity` of a barrier that other CTAs complete; bounded as
// mbar_wait_bounded, false when it ran out
__device__ __forceinline__ bool bmc_wait(uint64_t* bar, uint32_t parity, long long limit, int* status) {
    const long long t0 = clock64();
    for (;;) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(smem_addr(bar)), "r"(parity)
            : "memory");
        if (done) return true;
        if (clock64() - t0 > limit) {
            if (status) atomicExch(status, TFHE_STATUS_WAIT_TIMEOUT);
            return false;
        }
    }
}

// After a wait that ran out: stores of other CTAs may still be on their way
// into this CTA's shared memory although none is issued any more (a cluster
// barrier lies behind), so the CTA stays for a few thousand times their latency
// (about 1 ms)
__device__ __forceinline__ void bmc_drain() {
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000LL) {
    }
}

// LOST: the first CTA keeps back the digits of group 1 that the last one waits
// for (the probe of what the kernel does then)
template <int L, int T, int C, bool REF, bool LOST = false>
__global__ void __launch_bounds__(BM_THREADS, 1) br_mma_cluster_kernel(const BrArgs args) {
    using S = BmcShape<L, C>;
    constexpr int LOGN = 10, LOGH = 9, P = 2 * L, K = BM_K, M = 4 * T;
    constexpr int N = BM_N, H = BM_H, PPC = S::PPC, NA = S::NA, ND = S::ND;
    using PL = Plan<LOGH>;
    static_assert(C == 2 || C == 4 || C == 8, "clusters of two, four or eight CTAs");

    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2* dig = reinterpret_cast<double2*>(smem_raw);            // [ND][H]
    double2* out = C == 2 ? dig : dig + (size_t)ND * H;              // [NA][H] (C = 2: in dig)
    double2* rec = dig + (size_t)(ND + S::OUT) * H;                  // [K][P][PPC]: all digits of the CTA's points
    double2* stage = rec + (size_t)K * P * PPC;                      // [16 warps][STAGED][T][L][32]
    double2* gather = stage + (size_t)16 * S::STAGED * T * L * 32;   // ASYNC: [K][2][PPC] results of this CTA's points
    double2* hc = gather + S::GATHER;                       // exp(-i pi r / N), r < N
    double2* tw = hc + N;                                            // PL::TW
    double2* node = tw + PL::TW;                                     // [8] then [8][8] nodes, 4 factors each
    uint16_t* rot = reinterpret_cast<uint16_t*>(node + (8 + 64) * BM_NODE);   // [BM_ROT_GROUPS][K][M]
    uint64_t* bars = reinterpret_cast<uint64_t*>(rot + BM_ROT_GROUPS * K * M);   // digits, outputs
    int* bexp = reinterpret_cast<int*>(bars + 2);                    // NC

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = (int)cluster_rank();
    const long long cl = cluster_index_x(), ncl = cluster_count_x();
    const long long nsets = (args.B + K - 1) / K;
    const long long my_sets = cl < nsets ? (nsets - cl + ncl - 1) / ncl : 0;

    auto zeta = [&](int r) {                                         // zeta^r, 0 <= r < N, from the quarter table
        const double2 w = args.qt[r & (N / 2 - 1)];
        return r < N / 2 ? w : c_mul_mi(w);
    };
    for (int i = tid; i < N; i += BM_THREADS) hc[i] = zeta(i);
    for (int i = tid; i < PL::TW; i += BM_THREADS) tw[i] = args.tw[i];
    for (int i = tid; i < 8 + 64; i += BM_THREADS) {
        // node exponent E: below path bits b1 b2 b3 (b4 b5 b6), first level first
        const int depth = i < 8 ? 3 : 6, path = i < 8 ? i : i - 8;
        int E = N >> (depth + 1);
        for (int d = 1; d <= depth; ++d)
            if ((path >> (depth - d)) & 1) E += N >> (depth - d);
        node[i * 4 + 0] = zeta(E / 2);
        node[i * 4 + 1] = zeta(E / 4);
        node[i * 4 + 2] = zeta(E / 8);
        node[i * 4 + 3] = zeta(E / 8 + N / 4);
    }
    if (tid == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        mbar_fence_init();
    }
    cluster_barrier();                                               // tables and barriers ready, every CTA has started
    // bytes that reach this CTA per group
    constexpr uint32_t DIGIT_BYTES = K * P * PPC * sizeof(double2), OUT_BYTES = NA * H * sizeof(double2);

    // element e of local polynomial pq with exclusive-or x (2 k + a of it)
    auto at = [](int pq, int x, int e) { return pq * H + (e ^ ((e >> 3) & 7) ^ x); };
    // digit polynomial (k, bc) and output polynomial (k, a) of this CTA
    auto dig_poly = [](int k, int bc) { return C == 8 ? bc >> 1 : k * P + bc; };
    auto out_poly = [](int k, int a) { return C == 2 ? k * P + a : (C == 4 ? a : 0); };

    // outer pass: ciphertext k, polynomial a, points c + 64 n; level olv (LP)
    const int oc = tid & 63;
    const int oa = C == 8 ? (rank & 1) : (tid >> 6) & 1;
    const int ok = C == 2 ? (tid >> 7) & 1 : 0;
    const int olv = C == 4 ? tid >> 7 : tid >> 6;
    const bool owner = S::LP ? olv < L : tid < 256;
    const int ct_in = C == 2 ? 2 * rank + ok : (C == 4 ? rank : rank >> 1);   // of the cluster's four
    // inner passes: groups of 8 lanes, one block of one polynomial each
    const int t8 = lane & 7, grp = warp * 4 + (lane >> 3);
    // contraction: this warp's points, B and T as br_mma_kernel
    constexpr int PPW = PPC / 16;
    const int p0 = rank * PPC + warp * PPW;
    const int bk = lane >> 3, bdig = (lane >> 1) & 1, bcomp = (lane & 1) ^ ((lane >> 2) & 1);
    const int bsign = ((lane & 1) && !((lane >> 2) & 1)) ? 0x80000000 : 0;
    const int bx = bk * 2 + bdig;
    const double* bbase = reinterpret_cast<const double*>(rec + (bk * P + bdig) * PPC) + bcomp;
    const int to = lane >> 4, tm = (lane >> 2) & 3, tk = lane & 3;
    // where this lane's results go: output (ciphertext tk, polynomial to)
    const int out_rank = C == 2 ? tk >> 1 : (C == 4 ? tk : 2 * tk + to);
    const int out_x = C == 2 ? (tk & 1) * 2 + to : to;
    const uint32_t out_base = peer_smem(out + (size_t)out_poly(C == 2 ? tk & 1 : 0, to) * H, (uint32_t)out_rank) +
                              ((lane >> 2) & 1) * (uint32_t)sizeof(double);

    const double q = ldexp(1.0, args.log2_q);
    const double inv_q = ldexp(1.0, -args.log2_q);
    const double beta = ldexp(1.0, args.log2_beta);
    const double inv_qb = ldexp(1.0, args.log2_beta - args.log2_q);

    // key words of four points (two pairs) of group g
    constexpr int STEP = T * L * 32;                                 // double2 per pair of points
    const double2* key0 = reinterpret_cast<const double2*>(args.bsk_mma +
                                                           bm_key_at(L, T, 0, p0 >> 5, (p0 & 31) >> 1, 0, 0, lane, 0));
    constexpr size_t GROUP = (size_t)16 * 16 * STEP;                 // double2 per group
    auto load = [&](double2 (&kw)[T][L], int g, int u) {
#pragma unroll
        for (int t = 0; t < T; ++t)
#pragma unroll
            for (int s = 0; s < L; ++s) kw[t][s] = __ldg(key0 + (size_t)g * GROUP + u * STEP + (t * L + s) * 32);
    };
    // the first STAGED pairs of group g into this lane's shared-memory slots
    double2* slot = stage + (size_t)warp * S::STAGED * STEP + lane;
    auto copy = [&](int g) {
#pragma unroll
        for (int x = 0; x < S::STAGED * T * L; ++x)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(slot + x * 32)),
                         "l"(key0 + (size_t)g * GROUP + x * 32)
                         : "memory");
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto staged = [&](double2 (&kw)[T][L], int u) {
#pragma unroll
        for (int t = 0; t < T; ++t)
#pragma unroll
            for (int s = 0; s < L; ++s) kw[t][s] = slot[u * STEP + (t * L + s) * 32];
    };

    uint32_t phase = 0;                                              // of both barriers, one per group
    // A wait that runs out ends the CTA's loop with its group, by a vote at one of
    // the group's barriers: the others' waits for the next digits run out too, so a
    // cluster ends within a few limits.  A CTA that leaves writes no outputs; those
    // of a call that records a timeout are undefined all the same.  The vote is at
    // the barrier behind the results' wait for C = 8 and at the one behind the
    // contraction for C = 4, each where it costs nothing (n=630, us, no vote / behind
    // the results / behind the contraction: 32 ciphertexts 1142 / 1092 / 1156, 100
    // ciphertexts 1889 / 1940 / 1890).
    constexpr bool VOTE_LATE = C == 8;
    bool came = true, lost = false;
    for (long long iter = 0; iter < my_sets && !lost; ++iter) {
        const long long ct0 = (cl + iter * ncl) * K;
        double acc_lo[8], acc_hi[8];
        {
            const long long oct = min(ct0 + ct_in, args.B - 1);
            if constexpr (REF) {
                const int64_t* src = args.ct_init + oct * args.ct_stride + oa * N;
#pragma unroll
                for (int n = 0; n < 8; ++n) {
                    acc_lo[n] = (double)src[oc + 64 * n];
                    acc_hi[n] = (double)src[oc + 64 * n + H];
                }
            } else {
                const uint32_t* src = args.lut + oct * args.lut_stride + oa * N;
#pragma unroll
                for (int n = 0; n < 8; ++n) {
                    acc_lo[n] = (double)(int32_t)src[oc + 64 * n];
                    acc_hi[n] = (double)(int32_t)src[oc + 64 * n + H];
                }
            }
        }
        copy(0);

        for (int g = 0; g < args.G; ++g, phase ^= 1) {
            if (S::ASYNC && tid == 0) {
                mbar_arrive_expect_tx(&bars[0], DIGIT_BYTES);
                mbar_arrive_expect_tx(&bars[1], OUT_BYTES);
            }
            // the next group's key block into L2 (all CTAs together: each its share)
            if (tid == 0 && g + 1 < args.G && args.l2_prefetch) {
                const size_t block = (size_t)2 * P * M * H * sizeof(double2);
                const size_t share = ((block / gridDim.x) + 255) & ~(size_t)255;
                const size_t off = (size_t)blockIdx.x * share;
                if (off < block) {
                    const size_t len = min(share, block - off);
                    const char* base = reinterpret_cast<const char*>(args.bsk_mma + (size_t)(g + 1) * 4 * P * M * H);
                    prefetch_l2_bulk(base + off, (uint32_t)len);
                }
            }
            // rotation indices of the next BM_ROT_GROUPS groups of all four
            // ciphertexts (br_fp64_kernel's formula)
            if (g % BM_ROT_GROUPS == 0) {
                const int ng = min(BM_ROT_GROUPS, args.G - g);
                for (int x = tid; x < ng * K * M; x += BM_THREADS) {
                    const int gg = x / (K * M), k = (x / M) % K, m = x % M;
                    const long long ct = min(ct0 + k, args.B - 1);
                    if constexpr (REF) {
                        rot[x] = (uint16_t)(args.indices[(ct * args.G + g + gg) * M + m] & (2 * N - 1));
                        continue;
                    }
                    double v = 0.0;
                    const uint32_t* a = args.lwe_a + ct * args.lwe_n + (long long)(g + gg) * args.collapse;
                    for (int c = 0; c < args.collapse; ++c)
                        if ((m >> (args.collapse - 1 - c)) & 1) v += (double)(int32_t)a[c];
                    const double idx = rint((2.0 * N * v) / (q * args.n_lut)) * args.n_lut;
                    const int ri = (int)idx % (2 * N);
                    rot[x] = (uint16_t)(ri < 0 ? ri + 2 * N : ri);
                }
            }

            // outer pass: gadget digits, fold, the tree's first three levels
            if (owner) {
                double2 w[4];
                w[0] = make_double2(0.70710678118654752440, -0.70710678118654752440);   // zeta^(N/4)
                w[1] = make_double2(0.92387953251128675613, -0.38268343236508977173);   // zeta^(N/8)
                w[2] = make_double2(0.98078528040323044913, -0.19509032201612826785);   // zeta^(N/16)
                w[3] = make_double2(0.55557023301960222474, -0.83146961230254523708);   // zeta^(5N/16)
                double2 v[8];
                if constexpr (S::LP) {
#pragma unroll
                    for (int lvl = 0; lvl < L; ++lvl)
                        if (lvl <= olv) {
                            const double sc = lvl == 0 ? inv_qb : beta;
#pragma unroll
                            for (int n = 0; n < 8; ++n) {
                                const double lo = bm_rint(acc_lo[n], sc), hi = bm_rint(acc_hi[n], sc);
                                acc_lo[n] = fma(acc_lo[n], sc, -lo);
                                acc_hi[n] = fma(acc_hi[n], sc, -hi);
                                v[n] = make_double2(lo, -hi);
                            }
                        }
                    bm_forward8(v, w);
#pragma unroll
                    for (int n = 0; n < 8; ++n) dig[at(dig_poly(0, olv * 2 + oa), oa, oc + 64 * n)] = v[n];
                } else {
#pragma unroll
                    for (int lvl = 0; lvl < L; ++lvl) {
                        const double sc = lvl == 0 ? inv_qb : beta;
#pragma unroll
                        for (int n = 0; n < 8; ++n) {
                            const double lo = bm_rint(acc_lo[n], sc), hi = bm_rint(acc_hi[n], sc);
                            acc_lo[n] = fma(acc_lo[n], sc, -lo);
                            acc_hi[n] = fma(acc_hi[n], sc, -hi);
                            v[n] = make_double2(lo, -hi);
                        }
                        bm_forward8(v, w);
#pragma unroll
                        for (int n = 0; n < 8; ++n) dig[at(dig_poly(ok, lvl * 2 + oa), ok * 2 + oa, oc + 64 * n)] = v[n];
                    }
                }
            }
            __syncthreads();

            // inner passes, the last level into the owner of the block's points
#pragma unroll 1
            for (int task = grp; task < ND * 8; task += 64) {
                const int pq = task >> 3, blk = task & 7;
                const int k = C == 2 ? pq / P : 0;
                const int bc = C == 2 ? pq % P : (C == 4 ? pq : pq * 2 + oa);
                const int x = k * 2 + (bc & 1);
                double2 w[4], v[8];
#pragma unroll
                for (int i = 0; i < 4; ++i) w[i] = node[blk * 4 + i];
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = dig[at(pq, x, blk * 64 + t8 + 8 * j)];
                bm_forward8(v, w);
#pragma unroll
                for (int j = 0; j < 8; ++j) dig[at(pq, x, blk * 64 + t8 + 8 * j)] = v[j];
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 4; ++i) w[i] = node[(8 + blk * 8 + t8) * 4 + i];
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = dig[at(pq, x, blk * 64 + 8 * t8 + j)];
                bm_forward8(v, w);
#pragma unroll
                for (int j = 0; j < 8; ++j) dig[at(pq, x, blk * 64 + 8 * t8 + j)] = v[j];
                __syncwarp();
                // the warp's four blocks to their owners, 512 bytes in a row per
                // store (16-byte pieces of scattered rows take four times as long)
                const int kc = C == 2 ? 2 * rank + k : ct_in;
                const int x2 = kc * 2 + (bc & 1);
                const int blk0 = blk & 4;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int bi = blk0 + (i >> 1), e = (i & 1) * 32 + lane, eo = (bi % NA) * 64 + e;
                    const uint32_t dst = peer_smem(rec + (size_t)(kc * P + bc) * PPC + (eo ^ ((eo >> 3) & 7) ^ x2),
                                                   (uint32_t)(bi / NA));
                    const double2 z = dig[at(pq, x, bi * 64 + e)];
                    if constexpr (LOST)
                        if (g == 1 && rank == 0 && bi / NA == C - 1) continue;
                    if constexpr (S::ASYNC) st_async(dst, z, peer_smem(&bars[0], (uint32_t)(bi / NA)));
                    else st_peer(dst, z);
                }
            }
            double2 ka[T][L], kb[T][L];
            if constexpr (S::STAGED < 1) load(ka, g, 0);
            if constexpr (S::STAGED < 2) load(kb, g, 1);
            // every digit of this CTA's points is here
            if constexpr (S::ASYNC) came = bmc_wait(&bars[0], phase, args.wait_limit, args.status);
            else cluster_barrier();

            // contraction of this warp's points, four at a time
            {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
                if constexpr (S::STAGED >= 1) staged(ka, 0);
                if constexpr (S::STAGED >= 2) staged(kb, 1);
                int rr[T];
                const uint16_t* rg = rot + (g % BM_ROT_GROUPS) * K * M + tk * M + tm;
#pragma unroll
                for (int t = 0; t < T; ++t) rr[t] = rg[4 * t];
#pragma unroll 1
                for (int i0 = 0; i0 < PPW; i0 += 4) {
                    double c[4][T][2], b[4][L], y[2];
                    double2 w[T][2];
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int s = 0; s < L; ++s) {
                            const int e = warp * PPW + i0 + i;
                            const double x = bbase[(size_t)(2 * s * PPC + (e ^ ((e >> 3) & 7) ^ bx)) * 2];
                            b[i][s] = __hiloint2double(__double2hiint(x) ^ bsign, __double2loint(x));
                        }
                    bm_twist<T>(w, rr, hc, p0 + i0);
                    bm_products<L, T>(c, ka, kb, b, [&](int h) {
                        if (i0 + 4 < PPW) {
                            if (h == 0) load(ka, g, (i0 >> 1) + 2);
                            else load(kb, g, (i0 >> 1) + 3);
                        }
                    });
                    if (i0 == 0 && g + 1 < args.G) copy(g + 1);
                    bm_sums<T>(y, c, w, rr, lane);
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const int p = p0 + i0 + 2 * j + ((lane >> 3) & 1);
                        if constexpr (S::ASYNC) {
                            const int e = p - rank * PPC;
                            reinterpret_cast<double*>(gather + (tk * 2 + to) * PPC + (e ^ ((e >> 3) & 7) ^ (tk * 2 + to)))[(lane >> 2) & 1] = y[j];
                        } else {
                            st_peer(out_base + (uint32_t)((p ^ ((p >> 3) & 7) ^ out_x) * sizeof(double2)), y[j]);
                        }
                    }
                }
            }
            // every point of this CTA's outputs is here
            if constexpr (S::ASYNC) {
                if constexpr (VOTE_LATE) __syncthreads();
                else lost = __syncthreads_or(!came);
#pragma unroll
                for (int i = 0; i < 8 * PPC / BM_THREADS; ++i) {
                    const int o = (tid + i * BM_THREADS) / PPC, e = (tid + i * BM_THREADS) % PPC, p = rank * PPC + e;
                    const int k = o >> 1, a = o & 1, dst_rank = C == 4 ? k : 2 * k + a;
                    st_async(peer_smem(out + (size_t)out_poly(0, a) * H + (p ^ ((p >> 3) & 7) ^ a), (uint32_t)dst_rank),
                             gather[o * PPC + (e ^ ((e >> 3) & 7) ^ o)], peer_smem(&bars[1], (uint32_t)dst_rank));
                }
                came &= bmc_wait(&bars[1], phase, args.wait_limit, args.status);
            } else {
                cluster_barrier();
            }

            // inverse inner passes
            if (grp < NA * 8) {
                const int oq = grp >> 3, blk = grp & 7;
                const int k = C == 2 ? oq >> 1 : 0, a = C == 8 ? oa : oq & 1;
                double2* poly = out;
                const int pq = out_poly(k, a), x2 = k * 2 + a;
                double2 v[8], x[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) x[j] = poly[at(pq, x2, blk * 64 + 8 * t8 + j)];
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = x[bm_rev3(j)];
                dft8<true>(v);
#pragma unroll
                for (int j = 0; j < 8; ++j) poly[at(pq, x2, blk * 64 + 8 * t8 + j)] = v[j];
                __syncwarp();
#pragma unroll
                for (int j = 0; j < 8; ++j) x[j] = poly[at(pq, x2, blk * 64 + t8 + 8 * j)];
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = x[bm_rev3(j)];
                twiddle<8, 8, true>(v, tw + PL::tw_offset(1), t8);
                dft8<true>(v);
#pragma unroll
                for (int j = 0; j < 8; ++j) poly[at(pq, x2, blk * 64 + t8 + 8 * j)] = v[j];
            }
            if constexpr (VOTE_LATE) lost = __syncthreads_or(!came);
            else __syncthreads();

            // last superstage, untwist, round, centred reduction (every level's threads)
            if (owner) {
                double2 v[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = out[at(out_poly(ok, oa), ok * 2 + oa, oc + 64 * bm_rev3(j))];
                twiddle<8, 64, true>(v, tw, oc);
                dft8<true>(v);
#pragma unroll
                for (int n = 0; n < 8; ++n) {
                    const double2 u = c_mul(c_conj(hc[oc + 64 * n]), v[n]);
                    const double rlo = rint(u.x);
                    const double rhi = rint(-u.y);
                    acc_lo[n] = fma(-q, bm_rint(rlo, inv_q), rlo);
                    acc_hi[n] = fma(-q, bm_rint(rhi, inv_q), rhi);
                }
            } else {
                // written on every path, so nothing is held between here and there
#pragma unroll
                for (int n = 0; n < 8; ++n) acc_lo[n] = acc_hi[n] = 0.0;
            }
            if (S::ASYNC && lost) break;
        }
        if (lost) break;
        if constexpr (S::ASYNC && !VOTE_LATE) {
            lost = __syncthreads_or(!came);
            if (lost) break;
        } else {
            __syncthreads();                                         // dig and out are reused below
        }

        if constexpr (REF) {
            if (owner && (!S::LP || olv == 0) && ct0 + ct_in < args.B) {
                int64_t* dst = args.out_i64 + (ct0 + ct_in) * 2 * N + oa * N;
#pragma unroll
                for (int n = 0; n < 8; ++n) {
                    dst[oc + 64 * n] = __double2ll_rn(acc_lo[n]);
                    dst[oc + 64 * n + H] = __double2ll_rn(acc_hi[n]);
                }
            }
            continue;
        }
        // epilogue: rotate by -b~ and extract, as br_fp64_kernel; C = 8: the
        // CTA of polynomial 0 the masks, that of polynomial 1 the bodies
        uint32_t* acc = reinterpret_cast<uint32_t*>(smem_raw);       // [NA][N]
        if (owner && (!S::LP || olv == 0)) {
            uint32_t* dst = acc + (size_t)(C == 8 ? 0 : ok * 2 + oa) * N;
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                dst[oc + 64 * n] = (uint32_t)(long long)acc_lo[n];
                dst[oc + 64 * n + H] = (uint32_t)(long long)acc_hi[n];
            }
        }
        const int first = C == 2 ? 2 * rank : ct_in;                 // this CTA's first ciphertext of the four
        if (tid < S::NC) {
            const double b = (double)(int32_t)args.lwe_b[min(ct0 + first + tid, args.B - 1)];
            bexp[tid] = (int)(rint((2.0 * N * b) / (q * args.n_lut)) * args.n_lut);
        }
        __syncthreads();
        const int nl = args.n_lut;
        for (int k = 0; k < S::NC; ++k) {
            const long long ct = ct0 + first + k;
            if (ct >= args.B) break;
            const int bx2 = bexp[k];
            const uint32_t* mask = acc + (size_t)(C == 8 ? 0 : 2 * k) * N;
            const uint32_t* body = C == 8 ? acc : mask + N;
            const bool do_mask = C != 8 || oa == 0, do_body = C != 8 || oa == 1;
            if (args.acc_out)
                for (int i = tid; i < N; i += BM_THREADS) {
                    if (do_mask) args.acc_out[ct * 2 * N + i] = ncoef<LOGN>(mask, i + bx2);
                    if (do_body) args.acc_out[ct * 2 * N + N + i] = ncoef<LOGN>(body, i + bx2);
                }
            if (args.out_a && do_mask)
                for (int x = tid; x < nl * N; x += BM_THREADS) {
                    const int al = x / N, j = x % N;
                    args.out_a[ct * nl * N + x] = ncoef<LOGN>(mask, al - j + bx2);
                }
            if (args.out_b && do_body)
                for (int al = tid; al < nl; al += BM_THREADS) args.out_b[ct * nl + al] = ncoef<LOGN>(body, al + bx2);
        }
        __syncthreads();                                             // shared memory is reused by the next set
    }
    if (lost) asm volatile("cp.async.wait_group 0;" ::: "memory");
    cluster_barrier();
    if (lost) bmc_drain();
}

}  // namespace tfhe
