// Blind rotation at N = 2048, l_bs = 2 for small batches: two ciphertexts per
// cluster of four CTAs, outputs bit-identical to br_fp64_kernel.
//
// One ciphertext per cluster pair (br_split_kernel) pulls half of a group's key
// through each SM for that one ciphertext, half of its 17k cycles a group.  Here
// as many SMs serve a ciphertext, but CTA r transforms one polynomial of one of
// the two and contracts a quarter of the points for both, so an SM reads a
// quarter of the key and each word serves two ciphertexts.
//
// The spectrum's 1024 positions k0 128 + k1 16 + k2 (superstages 8.8.16) are cut
// into eight blocks w = (k0 / 2, k1 mod 2), 128 positions each (warp_pos); CTA r
// owns blocks 2 r and 2 r + 1, 256 of the key's slots in a row.  A radix-16
// butterfly lies inside a block, so:
//   forward: outer radix-8 pass and second superstage as the other kernels, then
//     a warp that owns two k0's runs their radix-16 butterflies, two lanes each
//     (a lane takes the even or the odd outputs: the first level's sums or
//     differences, and the three levels below them), and sends every point to
//     its block's owner;
//   contraction in the owner: a thread takes one point of one output for both
//     ciphertexts;
//   inverse: the radix-16 butterflies (four lanes each) still in the owner, which
//     sends their points to the polynomial's CTA; the other two superstages there.
// Every butterfly and sum has the operations of br_fp64_kernel in its order.
//
// Exchange: st.async stores counted on an mbarrier of the receiver, eight lanes
// 128 bytes in a row (j = (k0 mod 2) 4 + k1 / 2 the fastest index, exclusive-or
// of it with the row's low bits keeps the receiver's reads free of bank
// conflicts), one wait each for digits and outputs per group.  The key words of
// two patterns of the next group come by bulk copies while the inverse and the
// next forward transform run.
//
// n=742 with the key switch, ms: 37 ciphertexts 2.43, 64 2.53 (cluster pair
// 3.08).  About 13k cycles a group, a quarter of them the contraction; the rest
// is the chain of passes (the last and first superstages 3.4k on eight warps, the
// middle ones 2.2k) and the two exchanges (FP64 pipe 30%).  Four ciphertexts per cluster of eight took 2.50 ms, but
// only 14 such clusters are resident; four per cluster of four 4.47 ms.
//
// No buffer is written early: a CTA sends digits of group g + 1 only after all its
// outputs of group g have come, to which every CTA contributes after a barrier
// behind its contraction, the last reader of the digits; outputs of g + 1 come
// only from CTAs that hold all digits of g + 1, among them this CTA's own,
// sent behind a barrier after its last reads of the outputs of group g.  No
// thread misses a phase for the same reasons.
#pragma once

#include "br_cluster.cuh"
#include "br_mma_cluster.cuh"

namespace tfhe {

constexpr int BS_THREADS = 512;
constexpr int BS_C = 4, BS_K = 2;                    // CTAs and ciphertexts of a cluster
constexpr int BS_NB = 8 / BS_C;                      // blocks of 128 points per CTA
constexpr int BS_STAGED = 2;                         // patterns whose key words are copied ahead
constexpr int BS_ROT_GROUPS = 32;

// shared memory: staged key words, digit spectra, outputs, received digits,
// results, root and twiddle tables, barriers, rotation indices, b~
inline size_t br_share_smem(int M) {
    return (size_t)(BS_STAGED * 4 * BS_NB * 256 + (2 + 1) * 1024 + BS_NB * BS_K * 4 * 128 + BS_NB * BS_K * 2 * 128 +
                    1024 + Plan<10>::TW) * sizeof(double2) +
           (size_t)BS_ROT_GROUPS * M * BS_K * sizeof(uint16_t) + 3 * sizeof(uint64_t) + 2 * sizeof(int) + 16;
}

// outputs 2 kk + h of a 16-point DFT in r[bitrev3(kk)] (dft16's operations):
// in(n) the n-th input
template <bool INV, class In>
__device__ __forceinline__ void bs_half16(double2 (&r)[8], int h, In in) {
    const double s = h ? -1.0 : 1.0;                 // a + b or a - b
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const double2 a = in(j), b = in(j + 8);
        r[j] = make_double2(fma(s, b.x, a.x), fma(s, b.y, a.y));
    }
    if (h) {
#pragma unroll
        for (int j = 1; j < 8; ++j) {
            if (j == 4) r[j] = INV ? c_mul_pi(r[j]) : c_mul_mi(r[j]);
            else r[j] = c_mul(r[j], w16(j, INV));
        }
    }
#pragma unroll
    for (int half = 4; half >= 1; half >>= 1)
#pragma unroll
        for (int blk = 0; blk < 8; blk += 2 * half)
#pragma unroll
            for (int j = 0; j < half; ++j) {
                const double2 a = r[blk + j], b = r[blk + j + half];
                r[blk + j] = c_add(a, b);
                const double2 d = c_sub(a, b);
                const int m = j * (8 / half);
                if (m == 0) r[blk + j + half] = d;
                else if (m == 4) r[blk + j + half] = INV ? c_mul_pi(d) : c_mul_mi(d);
                else r[blk + j + half] = c_mul(d, w16(m, INV));
            }
}

// outputs 4 kk + 2 h2 + h in r[bitrev2(kk)]
template <bool INV, class In>
__device__ __forceinline__ void bs_quarter16(double2 (&r)[4], int h, int h2, In in) {
    const double s = h ? -1.0 : 1.0, s2 = h2 ? -1.0 : 1.0;
    double2 x[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const double2 a = in(j), b = in(j + 8);
        x[j] = make_double2(fma(s, b.x, a.x), fma(s, b.y, a.y));
    }
    if (h) {
#pragma unroll
        for (int j = 1; j < 8; ++j) {
            if (j == 4) x[j] = INV ? c_mul_pi(x[j]) : c_mul_mi(x[j]);
            else x[j] = c_mul(x[j], w16(j, INV));
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) r[j] = make_double2(fma(s2, x[j + 4].x, x[j].x), fma(s2, x[j + 4].y, x[j].y));
    if (h2) {
#pragma unroll
        for (int j = 1; j < 4; ++j) {
            if (j == 2) r[j] = INV ? c_mul_pi(r[j]) : c_mul_mi(r[j]);
            else r[j] = c_mul(r[j], w16(2 * j, INV));
        }
    }
#pragma unroll
    for (int half = 2; half >= 1; half >>= 1)
#pragma unroll
        for (int blk = 0; blk < 4; blk += 2 * half)
#pragma unroll
            for (int j = 0; j < half; ++j) {
                const double2 a = r[blk + j], b = r[blk + j + half];
                r[blk + j] = c_add(a, b);
                const double2 d = c_sub(a, b);
                r[blk + j + half] = half == 2 && j == 1 ? (INV ? c_mul_pi(d) : c_mul_mi(d)) : d;
            }
}

// LOST as in br_mma_cluster_kernel
template <bool T64, bool LOST = false>
__global__ void __launch_bounds__(BS_THREADS, 1) br_share_kernel(const BrArgs args) {
    constexpr int LOGN = 11, LOGH = 10, N = 2048, H = 1024, P = 4, K = BS_K;
    constexpr int NB = BS_NB, MS = BS_STAGED;
    using PL = Plan<LOGH>;
    static_assert(PL::radix(0) == 8 && PL::radix(1) == 8 && PL::radix(2) == 16, "superstages 8.8.16");

    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int M = args.M;
    double2* stage = reinterpret_cast<double2*>(smem_raw);          // [MS][2 out][2][NB 128][2] key words
    double2* spec = stage + MS * 4 * NB * 256;                       // [2 levels][H]
    double2* outp = spec + 2 * H;                                    // [8 w][16 n][8 j]
    double2* rec = outp + H;                                         // [NB][K][P][16 k2][8 j]
    double2* gat = rec + NB * K * P * 128;                           // [NB][K][2][16 k2][8 j]
    double2* qt_s = gat + NB * K * 2 * 128;                          // N / 2, swizzled
    double2* tw = qt_s + N / 2;                                      // PL::TW
    uint64_t* bars = reinterpret_cast<uint64_t*>(tw + PL::TW);       // digits, outputs, key words
    uint16_t* rot = reinterpret_cast<uint16_t*>(bars + 3);           // [BS_ROT_GROUPS][K][M]
    int* bexp = reinterpret_cast<int*>(rot + BS_ROT_GROUPS * K * M);
    volatile int* gave_up = bexp + 2;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = (int)cluster_rank();
    const long long ct0 = (long long)cluster_index_x() * K;
    auto qtab = [&](int r) { return qt_s[qsw<LOGN>(r)]; };

    for (int i = tid; i < N / 2; i += BS_THREADS) qt_s[qsw<LOGN>(i)] = args.qt[i];
    for (int i = tid; i < PL::TW; i += BS_THREADS) tw[i] = args.tw[i];
    if (tid == 0) {
        for (int i = 0; i < 3; ++i) mbar_init(&bars[i], 1);
        mbar_fence_init();
        *gave_up = 0;
    }
    cluster_barrier();                                               // tables and barriers ready, every CTA has started
    constexpr uint32_t DIGIT_BYTES = NB * K * P * 128 * sizeof(double2), OUT_BYTES = H * sizeof(double2);

    const double q = ldexp(1.0, args.log2_q);
    const double inv_q = ldexp(1.0, -args.log2_q);
    const double beta = ldexp(1.0, args.log2_beta);
    const double inv_qb = ldexp(1.0, args.log2_beta - args.log2_q);

    // transforms: level lvl of polynomial oa of ciphertext ok, butterfly c
    const int c = tid & 127, lvl = tid >> 7;
    const bool owner = lvl < 2;
    const int oa = rank & 1, ok = rank >> 1;
    const long long oct = min(ct0 + ok, args.B - 1);
    auto out_at = [](int w, int n, int j) { return (w * 16 + n) * 8 + (j ^ (n & 7)); };
    // row k2 of block polynomial `poly`, column j
    auto rec_at = [](int poly, int k2, int j) { return (poly * 16 + k2) * 8 + (j ^ (k2 & 1) ^ ((k2 & 2) << 1)); };

    // contraction: this lane's point (slot u, block cb of this CTA), output co
    const int co = warp & 1, sl = (warp >> 1) * 32 + lane;
    const int u = rank * NB * 128 + sl;
    const int pos = warp_pos(u);
    const int ku = key_slot<LOGH>(pos, 2, T64);                      // in the slots of the CTA's blocks
    const int e = 4 * args.freq[pos] + 1;
    const int cb = sl >> 7, ck2 = pos & 15, cj = ((pos >> 7) & 1) * 4 + ((pos >> 5) & 3);

    // key words of the staged patterns of group g, 8 KB a copy
    const size_t GROUP = (size_t)2 * P * M * H;
    auto copy = [&](int g) {
        if (tid == 0) mbar_arrive_expect_tx(&bars[2], MS * 4 * NB * 256 * sizeof(double2));
        if (warp == 0) {
            __syncwarp();
            if (lane < MS * 4) {
                const int m = lane >> 2, oj = lane & 3;              // pattern; (output, digit pair)
                bulk_load(stage + (m * 4 + oj) * NB * 256,
                          args.bsk + (size_t)g * GROUP + ((size_t)oj * M + m) * H * 2 + (size_t)rank * NB * 256,
                          NB * 256 * sizeof(double2), &bars[2]);
            }
        }
    };

    double acc_lo[8], acc_hi[8];
#pragma unroll
    for (int n2 = 0; n2 < 8; ++n2) {
        acc_lo[n2] = acc_hi[n2] = 0.0;
        if (owner) {
            if constexpr (T64) {
                const long long* src = args.lut64 + oct * args.lut_stride + oa * N;
                acc_lo[n2] = (double)src[c + 128 * n2];
                acc_hi[n2] = (double)src[c + 128 * n2 + H];
            } else {
                const uint32_t* src = args.lut + oct * args.lut_stride + oa * N;
                acc_lo[n2] = (double)(int32_t)src[c + 128 * n2];
                acc_hi[n2] = (double)(int32_t)src[c + 128 * n2 + H];
            }
        }
    }
    copy(0);

    uint32_t phase = 0;                                              // of all barriers, one per group
    // a wait that runs out ends the loop with its group (see
    // br_mma_cluster_kernel)
    bool came = true, lost = false;
    for (int g = 0; g < args.G; ++g, phase ^= 1) {
        if (tid == 0) {
            mbar_arrive_expect_tx(&bars[0], DIGIT_BYTES);
            mbar_arrive_expect_tx(&bars[1], OUT_BYTES);
        }
        // a coming group's key block into L2 (all CTAs together: each its share)
        const int ahead = g + 2;
        if (tid == 0 && ahead < args.G && args.l2_prefetch) {
            const size_t block = GROUP * sizeof(double2);
            const size_t share = ((block / gridDim.x) + 255) & ~(size_t)255;
            const size_t off = (size_t)blockIdx.x * share;
            if (off < block)
                prefetch_l2_bulk(reinterpret_cast<const char*>(args.bsk + (size_t)ahead * GROUP) + off,
                                 (uint32_t)min(share, block - off));
        }
        // rotation indices of the next BS_ROT_GROUPS groups (br_fp64_kernel's
        // formulas); the last reader of the old ones is behind a barrier
        if (g % BS_ROT_GROUPS == 0) {
            const int ng = min(BS_ROT_GROUPS, args.G - g);
            for (int x = tid; x < ng * K * M; x += BS_THREADS) {
                const int gg = x / (K * M), k = (x / M) % K, m = x % M;
                const long long ct = min(ct0 + k, args.B - 1);
                if constexpr (T64) {
                    unsigned long long v = 0ULL;
                    const unsigned long long* a = args.lwe_a64 + ct * args.lwe_n + (long long)(g + gg) * args.collapse;
                    for (int i = 0; i < args.collapse; ++i)
                        if ((m >> (args.collapse - 1 - i)) & 1) v += a[i];
                    const int ln = __ffs(args.n_lut) - 1;
                    rot[x] = (uint16_t)((rne_div_pow2((long long)v, 63 - LOGN + ln) << ln) & (2 * N - 1));
                } else {
                    double v = 0.0;
                    const uint32_t* a = args.lwe_a + ct * args.lwe_n + (long long)(g + gg) * args.collapse;
                    for (int i = 0; i < args.collapse; ++i)
                        if ((m >> (args.collapse - 1 - i)) & 1) v += (double)(int32_t)a[i];
                    const double idx = rint((2.0 * N * v) / (q * args.n_lut)) * args.n_lut;
                    const int ri = (int)idx % (2 * N);
                    rot[x] = (uint16_t)(ri < 0 ? ri + 2 * N : ri);
                }
            }
        }

        // digits of this thread's level, fold and twist, first superstage
        double2* poly = spec + lvl * H;
        if (owner) {
            double2 v[8];
#pragma unroll
            for (int n2 = 0; n2 < 8; ++n2) {
                double ylo = acc_lo[n2] * inv_qb, dlo = rint(ylo);
                double yhi = acc_hi[n2] * inv_qb, dhi = rint(yhi);
                if (lvl) {
                    ylo = (ylo - dlo) * beta;
                    dlo = rint(ylo);
                    yhi = (yhi - dhi) * beta;
                    dhi = rint(yhi);
                }
                const double2 w = qtab(c + 128 * n2);
                v[n2] = make_double2(fma(w.x, dlo, w.y * dhi), fma(w.y, dlo, -w.x * dhi));
            }
            dft8<false>(v);
#pragma unroll
            for (int k2 = 1; k2 < 8; ++k2) v[k2] = c_mul(v[k2], tw[(k2 - 1) * 128 + c]);
#pragma unroll
            for (int k2 = 0; k2 < 8; ++k2) poly[swz(c + 128 * k2)] = v[k2];
        }
        __syncthreads();
        if (owner) {
            dif_stage<8, 16>(poly, tw + PL::tw_offset(1), c);
            __syncwarp();
            // radix 16 of this warp's two k0's, outputs of parity h
            const int wq = warp & 3, h = lane >> 4, kb = (lane >> 3) & 1, j = lane & 7;
            const int base = (2 * wq + (j >> 2)) * 128 + ((j & 3) * 2 + kb) * 16;
            double2 r[8];
            bs_half16<false>(r, h, [&](int n) { return poly[swz(base + n)]; });
            const int w = 2 * wq + kb;
            const uint32_t dst_rank = (uint32_t)(w / NB);
            const uint32_t dst = peer_smem(rec, dst_rank), bar = peer_smem(&bars[0], dst_rank);
            const int row = ((w % NB) * K + ok) * P + 2 * lvl + oa;
            const bool kept_back = LOST && g == 1 && rank == 0 && dst_rank == BS_C - 1;
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)
                if (!kept_back) st_async(dst + (uint32_t)(rec_at(row, 2 * kk + h, j) * sizeof(double2)), r[bm_rev3(kk)], bar);
        }
        // the next two patterns' key words are on their way during the waits
        const double2* kg = args.bsk + (size_t)g * GROUP + (size_t)co * 2 * M * H * 2 + 2 * (size_t)ku;
        double2 kw[2][P];
        auto load = [&](int m) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int jj = 0; jj < 2; ++jj) ldg_pair(kg + ((size_t)jj * M + m + i) * H * 2, kw[i][2 * jj], kw[i][2 * jj + 1]);
        };
        load(MS);
        // every digit of this CTA's points is here, and the staged key words
        came = mbar_wait_bounded(&bars[2], phase, args.wait_limit, args.status);
        came &= bmc_wait(&bars[0], phase, args.wait_limit, args.status);

        // contraction: out = sum_m X^{r_m} sum_bc BSK[g, o, bc, m] DEC[bc]
        {
            double2 d[K][P], s[K];
#pragma unroll
            for (int i = 0; i < K; ++i) {
                s[i] = make_double2(0.0, 0.0);
#pragma unroll
                for (int bc = 0; bc < P; ++bc) d[i][bc] = rec[rec_at((cb * K + i) * P + bc, ck2, cj)];
            }
            const uint16_t* rg = rot + (g % BS_ROT_GROUPS) * K * M;
            auto one = [&](int m, const double2 (&k)[P]) {
#pragma unroll
                for (int i = 0; i < K; ++i) {
                    double2 t = make_double2(0.0, 0.0);
#pragma unroll
                    for (int bc = 0; bc < P; ++bc) c_mac(t, k[bc], d[i][bc]);
                    c_mac(s[i], root2n<LOGN, true>(qt_s, rg[i * M + m] * e), t);
                }
            };
#pragma unroll
            for (int m = 0; m < MS; ++m) {
                double2 k[P];
#pragma unroll
                for (int x = 0; x < P; ++x) k[x] = stage[(m * 4 + co * 2 + (x >> 1)) * NB * 256 + 2 * (ku & (NB * 128 - 1)) + (x & 1)];
                one(m, k);
            }
#pragma unroll 1
            for (int m = MS; m < M; m += 2) {
                if (m > MS) load(m);
                one(m, kw[0]);
                one(m + 1, kw[1]);
            }
#pragma unroll
            for (int i = 0; i < K; ++i) gat[rec_at((cb * K + i) * 2 + co, ck2, cj)] = s[i];
        }
        if (g + 1 < args.G) {
            __syncthreads();
            fence_proxy_async_smem();
            copy(g + 1);
        } else {
            lost = __syncthreads_or(!came);
            if (lost) break;
        }

        // inverse radix 16 of this CTA's blocks, its points to the polynomials' CTAs
        if (warp < 8) {
            const int j = lane & 7, h = (lane >> 3) & 1, h2 = lane >> 4;
            const int b = warp >> 2, k = (warp >> 1) & 1, o = warp & 1;
            double2 r[4];
            bs_quarter16<true>(r, h, h2, [&](int n) { return gat[rec_at((b * K + k) * 2 + o, n, j)]; });
            const uint32_t dst_rank = (uint32_t)(2 * k + o);
            const uint32_t dst = peer_smem(outp, dst_rank), bar = peer_smem(&bars[1], dst_rank);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
                st_async(dst + (uint32_t)(out_at(rank * NB + b, 4 * kk + 2 * h2 + h, j) * sizeof(double2)),
                         r[((kk & 1) << 1) | (kk >> 1)], bar);
        }
        came = came && bmc_wait(&bars[1], phase, args.wait_limit, args.status);
        if (!came) *gave_up = 1;

        // inverse second superstage: butterfly (k0, n)
        if (lvl == 0) {
            double2* op = outp;
            const int k0 = c >> 4, n = c & 15;
            double2 v[8];
#pragma unroll
            for (int k1 = 0; k1 < 8; ++k1) v[k1] = op[out_at((k0 >> 1) * 2 + (k1 & 1), n, (k0 & 1) * 4 + (k1 >> 1))];
            twiddle<8, 16, true>(v, tw + PL::tw_offset(1), n);
            dft8<true>(v);
#pragma unroll
            for (int k1 = 0; k1 < 8; ++k1) op[out_at((k0 >> 1) * 2 + (k1 & 1), n, (k0 & 1) * 4 + (k1 >> 1))] = v[k1];
        }
        __syncthreads();
        const int ended = *gave_up;

        // last superstage, untwist, round, centred reduction (both levels' threads)
        if (owner) {
            const double2* op = outp;
            const int k1 = c >> 4, n = c & 15;
            double2 v[8];
#pragma unroll
            for (int k0 = 0; k0 < 8; ++k0) v[k0] = op[out_at((k0 >> 1) * 2 + (k1 & 1), n, (k0 & 1) * 4 + (k1 >> 1))];
            twiddle<8, 128, true>(v, tw, c);
            dft8<true>(v);
#pragma unroll
            for (int n2 = 0; n2 < 8; ++n2) {
                const double2 y = c_mul(c_conj(qtab(c + 128 * n2)), v[n2]);
                const double rlo = rint(y.x);
                const double rhi = rint(-y.y);
                acc_lo[n2] = rlo - q * rint(rlo * inv_q);
                acc_hi[n2] = rhi - q * rint(rhi * inv_q);
            }
        } else {
            // written on every path, so nothing is held between here and there
#pragma unroll
            for (int n2 = 0; n2 < 8; ++n2) acc_lo[n2] = acc_hi[n2] = 0.0;
        }
        lost = ended;
        if (lost) {
            if (g + 1 < args.G) phase ^= 1;                          // of the key words on their way
            break;
        }
    }

    if (lost) {
        // this CTA's own bulk copies land (or have landed) before it ends
        mbar_wait_bounded(&bars[2], phase, args.wait_limit, args.status);
        cluster_barrier();
        bmc_drain();
        return;
    }

    // epilogue: rotate by -b~ and extract, as br_cluster_kernel (the CTA of
    // polynomial 0 the masks, that of polynomial 1 the bodies).  The digit
    // spectra, which no peer touches, give way to the accumulator words; their
    // last readers are behind the barriers above.
    const bool valid = ct0 + ok < args.B;
    const int nl = args.n_lut;
    auto extract = [&](auto* acc, auto coef, auto* acc_out, auto* out_a, auto* out_b, int bx) {
        if (acc_out)
            for (int i = tid; i < N; i += BS_THREADS) acc_out[oct * 2 * N + oa * N + i] = coef(acc, i + bx);
        if (out_a && oa == 0)
            for (int x = tid; x < nl * N; x += BS_THREADS) {
                const int al = x / N, jx = x % N;
                out_a[oct * nl * N + x] = coef(acc, al - jx + bx);
            }
        if (out_b && oa == 1)
            for (int al = tid; al < nl; al += BS_THREADS) out_b[oct * nl + al] = coef(acc, al + bx);
    };
    if constexpr (T64) {
        typedef unsigned long long u64;
        u64* acc = reinterpret_cast<u64*>(spec);
        if (lvl == 0) {
#pragma unroll
            for (int n2 = 0; n2 < 8; ++n2) {
                acc[c + 128 * n2] = (u64)__double2ll_rn(acc_lo[n2]);
                acc[c + 128 * n2 + H] = (u64)__double2ll_rn(acc_hi[n2]);
            }
        }
        if (tid == 0) {
            const int ln = __ffs(nl) - 1;
            bexp[0] = (int)((rne_div_pow2((long long)args.lwe_b64[oct], 63 - LOGN + ln) << ln) & (2 * N - 1));
        }
        __syncthreads();
        if (valid)
            extract(acc, [](const u64* p, int i) { return ncoef64<LOGN>(p, i); }, args.acc_out64, args.out_a64,
                    args.out_b64, bexp[0]);
    } else {
        uint32_t* acc = reinterpret_cast<uint32_t*>(spec);
        if (lvl == 0) {
#pragma unroll
            for (int n2 = 0; n2 < 8; ++n2) {
                acc[c + 128 * n2] = (uint32_t)(long long)acc_lo[n2];
                acc[c + 128 * n2 + H] = (uint32_t)(long long)acc_hi[n2];
            }
        }
        if (tid == 0) {
            const double b = (double)(int32_t)args.lwe_b[oct];
            bexp[0] = (int)(rint((2.0 * N * b) / (q * nl)) * nl);
        }
        __syncthreads();
        if (valid)
            extract(acc, [](const uint32_t* p, int i) { return ncoef<LOGN>(p, i); }, args.acc_out, args.out_a, args.out_b,
                    bexp[0]);
    }
    cluster_barrier();
}

}  // namespace tfhe
