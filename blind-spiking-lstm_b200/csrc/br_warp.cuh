// Batched blind rotation at N = 2048, l_bs = 2, NP pairs of ciphertexts per CTA
// of 256 threads: the transforms' inner superstages and the key contraction
// stay inside a warp, and the digit spectra wait in tensor memory, so each key
// word loaded serves four ciphertexts.
//
// The radix-8.8.16 transform of H = 1024 points (Plan<10>) is cut at other
// places than its superstages, the butterflies and their operations being
// those of br_fp64_kernel (so every value, and the outputs, are
// bit-identical to it):
//   outer pass (all 256 threads, registers): the first radix-8 superstage and
//     the first radix-2 level of the second.  A thread owns the coefficients of
//     two of its butterflies, c and c + 64 (c < 64), of one polynomial; what is
//     left are 16 independent blocks of 64 points per polynomial;
//   inner pass (one warp, radix 16): the second superstage's other two levels,
//     its twiddles, and the first two levels of the radix-16 superstage.  Warp w
//     owns the blocks (first digit 2 (w / 2) + b, half w mod 2), b = 0, 1, of
//     all eight digit polynomials of the two ciphertexts: lane = (polynomial,
//     4 columns), block b in turn;
//   contraction (same warp, registers): a lane holds four neighbouring points
//     of all eight polynomials, finishes the radix-16 superstage (two levels)
//     and parks the spectra in its tensor-memory lane; when both pairs are
//     there it contracts point after point with the key and starts the inverse
//     transform (two levels), so neither the digit spectra nor the products
//     pass through shared memory between these steps; then the inverse inner
//     and outer passes.
// Shared memory holds the spectra of one pair at a time (128 KB), tensor
// memory those of both (256 KB, all of it).  Per group and ciphertext 384 KB
// pass through shared memory instead of the 576 KB of superstage after
// superstage, and a group has two CTA barriers per pair.
//
// What bounds it: FP64 issue.  A DFMA takes 2 cycles per warp and scheduler,
// 2.4 to 2.9 with three distinct register operands, which puts the floor of
// two ciphertexts' group (n=742: four patterns) at about 16k cycles; measured
// 22.9k, br_fp64_kernel with 16 warps and two ciphertexts per key word 25.9k
// (16384 ciphertexts 275 -> 240 ms); with eight patterns on the 64-bit torus
// 30.4k against 36.5k.  The FP64 pipe is 58% busy (50% before), the shared-memory
// pipe 57%.  Why four
// ciphertexts per key word: with all SMs in step a key word takes about 1100
// cycles from L2, so eight warps with the key words of two steps in flight
// draw 50 bytes per cycle; two ciphertexts per word would need twice that.
#pragma once

#include <type_traits>

#include "br_fp64.cuh"

namespace tfhe {

constexpr int BW_THREADS = 256;
constexpr uint32_t BW_TM_COLS = 512;

// slot of root r (0 <= r < N) in the shared-memory table of the half circle,
// one entry left out after every 128: a warp's consecutive roots (outer pass)
// and its X^r lookups (contraction: the lanes of a wavefront are r 128 apart)
// then fall in distinct bank groups for every odd r
constexpr int BW_ROOTS = 2048 + 2048 / 128;
__device__ __forceinline__ int bw_root(int r) { return r + (r >> 7); }

// shared memory of br_warp_kernel<.., NP>: one pair's digit spectra, the root
// and twiddle tables, the rotation indices of every group (16 bits each), b~
// and the tensor-memory address
inline size_t br_warp_smem(int NP, int G, int M) {
    const int N = 2048, H = N / 2;
    const size_t tables = (size_t)(BW_ROOTS + Plan<10>::TW + 16) * sizeof(double2);
    const size_t rot = (((size_t)2 * NP * G * M * sizeof(uint16_t)) + 15) & ~(size_t)15;
    return (size_t)2 * 4 * H * sizeof(double2) + tables + rot + 2 * NP * sizeof(int) + 32;
}

// 16 double2 <-> 64 words of this thread's tensor-memory lane, 32 at a time;
// the load waits for its own words
__device__ __forceinline__ void bw_tm_load(uint32_t taddr, double2 (&v)[8]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i)
        v[i] = make_double2(__hiloint2double((int)r[4 * i + 1], (int)r[4 * i]),
                            __hiloint2double((int)r[4 * i + 3], (int)r[4 * i + 2]));
}

__device__ __forceinline__ void bw_tm_store(uint32_t taddr, const double2 (&v)[8]) {
    uint32_t r[32];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        r[4 * i] = (uint32_t)__double2loint(v[i].x);
        r[4 * i + 1] = (uint32_t)__double2hiint(v[i].x);
        r[4 * i + 2] = (uint32_t)__double2loint(v[i].y);
        r[4 * i + 3] = (uint32_t)__double2hiint(v[i].y);
    }
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
        "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
        "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}

__device__ __forceinline__ void bw_tm_store_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// rint(x) for |x| < 2^51 (round half to even by adding and subtracting
// 1.5 2^52; the sign of a zero may differ, which no sum or product here keeps)
__device__ __forceinline__ double bw_rint_add(double x, double scale) {
    constexpr double MAGIC = 6755399441055744.0;
    return __dadd_rn(fma(x, scale, MAGIC), -MAGIC);
}

// element e of polynomial q in shared memory: the lanes of the outer pass
// (consecutive e), of the inner pass (4 columns of 8 polynomials) and of the
// contraction (every fourth e) all take the minimum of wavefronts
__device__ __forceinline__ int bw_at(int q, int e) { return q * 1024 + (e ^ ((e >> 3) & 3) ^ ((q & 1) << 2)); }

// forward inner pass of one block half h (h = 1: the differences of the
// second superstage's first level; uniform across the warp): v[4 x + u] is the point at span-16 index
// x (of 4) and column t + 4 u (of 16)
__device__ __forceinline__ void bw_inner_forward(double2 (&v)[16], int h, const double2* tw1, int t, double2 wa,
                                                 double2 wb, double2 wc) {
    constexpr double R2 = 0.70710678118654752440084436210485;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        // the levels of dft8<false> at spans 2 and 1 (points x, x + 4 h)
        // (products and the sums they enter in one branch: the compiler fuses
        // them there as it does in dft8)
        const double2 a0 = v[u];
        double2 b0, b1, b2, b3;
        if (h) {
            const double2 a1 = make_double2(R2 * (v[4 + u].x + v[4 + u].y), R2 * (v[4 + u].y - v[4 + u].x));
            const double2 a2 = c_mul_mi(v[8 + u]);
            const double2 a3 = make_double2(R2 * (v[12 + u].y - v[12 + u].x), -R2 * (v[12 + u].x + v[12 + u].y));
            b0 = c_add(a0, a2);
            b2 = c_sub(a0, a2);
            b1 = c_add(a1, a3);
            b3 = c_mul_mi(c_sub(a1, a3));
        } else {
            b0 = c_add(a0, v[8 + u]);
            b2 = c_sub(a0, v[8 + u]);
            b1 = c_add(v[4 + u], v[12 + u]);
            b3 = c_mul_mi(c_sub(v[4 + u], v[12 + u]));
        }
        v[u] = c_add(b0, b1);
        v[4 + u] = c_sub(b0, b1);
        v[8 + u] = c_add(b2, b3);
        v[12 + u] = c_sub(b2, b3);
        // W_128^(column k2), k2 = 0 4 2 6 (h = 0) or 1 5 3 7 (h = 1)
        const double2* w = tw1 + h * 16 + t + 4 * u;
        if (h) v[u] = c_mul(v[u], tw1[t + 4 * u]);
        v[4 + u] = c_mul(v[4 + u], w[3 * 16]);
        v[8 + u] = c_mul(v[8 + u], w[1 * 16]);
        v[12 + u] = c_mul(v[12 + u], w[5 * 16]);
    }
#pragma unroll
    for (int x = 0; x < 4; ++x) {
        // dft16's levels at half = 8 and 4; wa, wb, wc = w16(t), w16(t + 4), w16(2 t)
        double2* p = v + 4 * x;
        double2 s0 = c_add(p[0], p[2]), d0 = c_mul(c_sub(p[0], p[2]), wa);
        double2 s1 = c_add(p[1], p[3]), d1 = c_mul(c_sub(p[1], p[3]), wb);
        p[0] = c_add(s0, s1);
        p[1] = c_mul(c_sub(s0, s1), wc);
        p[2] = c_add(d0, d1);
        p[3] = c_mul(c_sub(d0, d1), wc);
    }
}

// inverse inner pass: dft16's last two levels, the conjugate twiddles and the
// first two levels of dft8<true>
__device__ __forceinline__ void bw_inner_inverse(double2 (&v)[16], int h, const double2* tw1, int t) {
    constexpr double R2 = 0.70710678118654752440084436210485;
#pragma unroll
    for (int x = 0; x < 4; ++x) {
        double2* p = v + 4 * x;
        const double2 s0 = c_add(p[0], p[1]), d0 = c_sub(p[0], p[1]);
        const double2 s1 = c_add(p[2], p[3]), d1 = c_mul_pi(c_sub(p[2], p[3]));
        p[0] = c_add(s0, s1);
        p[2] = c_sub(s0, s1);
        p[1] = c_add(d0, d1);
        p[3] = c_sub(d0, d1);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const double2* w = tw1 + h * 16 + t + 4 * u;
        double2 a0 = v[u];
        if (h) a0 = c_mul(a0, c_conj(tw1[t + 4 * u]));
        const double2 a4 = c_mul(v[4 + u], c_conj(w[3 * 16]));
        const double2 a2 = c_mul(v[8 + u], c_conj(w[1 * 16]));
        const double2 a6 = c_mul(v[12 + u], c_conj(w[5 * 16]));
        const double2 s0 = c_add(a0, a4), s2 = c_add(a2, a6);
        double2 d0 = c_sub(a0, a4), d2 = c_sub(a2, a6);
        // points b[0], b[4], b[2], b[6] (+ h) of dft8<true> at their places
        v[u] = c_add(s0, s2);
        if (h) {
            d0 = make_double2(R2 * (d0.x - d0.y), R2 * (d0.x + d0.y));
            d2 = make_double2(-R2 * (d2.x + d2.y), R2 * (d2.x - d2.y));
            v[4 + u] = c_add(d0, d2);
            v[8 + u] = c_mul_pi(c_sub(s0, s2));
            v[12 + u] = c_mul_pi(c_sub(d0, d2));
        } else {
            d2 = c_mul_pi(d2);
            v[4 + u] = c_add(d0, d2);
            v[8 + u] = c_sub(s0, s2);
            v[12 + u] = c_sub(d0, d2);
        }
    }
}

template <bool T64, int NP>
__global__ void __launch_bounds__(BW_THREADS, 1) br_warp_kernel(const BrArgs args) {
    constexpr int LOGN = 11, LOGH = 10, L = 2, P = 4, K = 2 * NP;
    constexpr int N = 1 << LOGN, H = N / 2, Q8 = H / 8;
    using PL = Plan<LOGH>;
    static_assert(PL::radix(0) == 8 && PL::radix(1) == 8 && PL::radix(2) == 16, "superstages 8.8.16");

    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int M = args.M;
    double2* dec = reinterpret_cast<double2*>(smem_raw);            // 2 * P * H: one pair
    double2* hc = dec + (size_t)2 * P * H;                           // exp(-i pi r / N), r < N, at bw_root(r)
    double2* tw = hc + BW_ROOTS;                                          // PL::TW
    double2* w16t = tw + PL::TW;                                     // 8: w16(m, false), 8: w16(m, true)
    uint16_t* rot = reinterpret_cast<uint16_t*>(w16t + 16);          // [G M][K]
    const int GM = args.G * M;
    int* bexp = reinterpret_cast<int*>(rot + ((K * GM + 7) & ~7));   // K
    uint32_t* tm_slot = reinterpret_cast<uint32_t*>(bexp + K);
    const double2* tw1 = tw + PL::tw_offset(1);
    auto qtab = [&](int r) { return hc[bw_root(r)]; };

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long nsets = (args.B + K - 1) / K;
    const long long my_sets = blockIdx.x < nsets ? (nsets - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tm_slot)),
                     "r"(BW_TM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    for (int i = tid; i < N / 2; i += BW_THREADS) {
        const double2 w = args.qt[i];
        hc[bw_root(i)] = w;
        hc[bw_root(i + N / 2)] = c_mul_mi(w);
    }
    for (int i = tid; i < PL::TW; i += BW_THREADS) tw[i] = args.tw[i];
    if (tid < 16) w16t[tid] = w16(tid & 7, tid >= 8);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tm_base = *tm_slot;
    // this thread's tensor-memory lane: 256 columns, pair p at 128 p, point s
    // of the contraction at 32 s
    const uint32_t tm = tm_base + ((uint32_t)(warp & 3) << 21) + (uint32_t)(warp >> 2) * 256;

    // outer pass: ciphertext k, polynomial a, butterflies c and c + 64
    const int ok = tid >> 7, oa = (tid >> 6) & 1, oc = tid & 63;
    // inner pass: columns t + 4 u of the warp's blocks of half wh
    const int wh = warp & 1, wk = warp & ~1;
    const int it = lane & 3;
    // contraction: block wk + cb, four points from index 4 cg
    const int cb = lane >> 4, cg = lane & 15;
    const int cbase = (wk + cb) * 128 + wh * 64 + 4 * cg;
    // evaluation point zeta^e of the lane's first point; the others' differ by
    // multiples of N / 2 (third digit's bits 3 and 2)
    const int e0 = 4 * args.freq[warp_pos(warp * 128 + lane)] + 1;
    const int jg = 2 * (cg & 1) + ((cg >> 1) & 1);

    const double q = ldexp(1.0, args.log2_q);
    const double inv_q = ldexp(1.0, -args.log2_q);
    const double beta = ldexp(1.0, args.log2_beta);
    const double inv_qb = ldexp(1.0, args.log2_beta - args.log2_q);

    // digits of one ciphertext's owned coefficients, fold + twist, first
    // superstage and one level more, into the pair's spectra
    auto outer_forward = [&](const double (&acc_lo)[2][8], const double (&acc_hi)[2][8]) {
        double2 v[2][L][8];
#pragma unroll
        for (int col = 0; col < 2; ++col) {
            const int on1 = oc + 64 * col;
#pragma unroll
            for (int n2 = 0; n2 < 8; ++n2) {
                const double2 w = qtab(on1 + Q8 * n2);   // zeta^i
                const double lo0 = bw_rint_add(acc_lo[col][n2], inv_qb), hi0 = bw_rint_add(acc_hi[col][n2], inv_qb);
                v[col][0][n2] = make_double2(fma(w.x, lo0, w.y * hi0), fma(w.y, lo0, -w.x * hi0));
                const double lo1 = bw_rint_add(fma(acc_lo[col][n2], inv_qb, -lo0), beta);
                const double hi1 = bw_rint_add(fma(acc_hi[col][n2], inv_qb, -hi0), beta);
                v[col][1][n2] = make_double2(fma(w.x, lo1, w.y * hi1), fma(w.y, lo1, -w.x * hi1));
            }
#pragma unroll
            for (int lvl = 0; lvl < L; ++lvl) dft8<false>(v[col][lvl]);
#pragma unroll
            for (int k2 = 1; k2 < 8; ++k2) {
                const double2 w = tw[(k2 - 1) * Q8 + on1];
#pragma unroll
                for (int lvl = 0; lvl < L; ++lvl) v[col][lvl][k2] = c_mul(v[col][lvl][k2], w);
            }
        }
#pragma unroll
        for (int lvl = 0; lvl < L; ++lvl)
#pragma unroll
            for (int k2 = 0; k2 < 8; ++k2) {
                const int qi = ok * P + lvl * 2 + oa;
                dec[bw_at(qi, oc + Q8 * k2)] = c_add(v[0][lvl][k2], v[1][lvl][k2]);
                dec[bw_at(qi, oc + 64 + Q8 * k2)] = c_sub(v[0][lvl][k2], v[1][lvl][k2]);
            }
    };

    // inner pass of the pair in shared memory (one block of one polynomial per
    // four lanes), then the last two levels, into tensor memory
    auto inner_forward = [&](int pair) {
        {
            const int qi = lane >> 2;
            const double2 wa = w16t[it], wb = w16t[it + 4], wc = w16t[2 * it];
            double2 v[2][16];
#pragma unroll
            for (int b = 0; b < 2; ++b)
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    v[b][j] = dec[bw_at(qi, (wk + b) * 128 + wh * 64 + it + 16 * (j >> 2) + 4 * (j & 3))];
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                bw_inner_forward(v[b], wh, tw1, it, wa, wb, wc);
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    dec[bw_at(qi, (wk + b) * 128 + wh * 64 + it + 16 * (j >> 2) + 4 * (j & 3))] = v[b][j];
            }
        }
        __syncwarp();
        double2 d[4][8];
#pragma unroll
        for (int x = 0; x < 8; ++x) {
            double2 y[4];
#pragma unroll
            for (int s = 0; s < 4; ++s) y[s] = dec[bw_at(x, cbase + s)];
            const double2 r0 = c_add(y[0], y[2]), r2 = c_sub(y[0], y[2]);
            const double2 r1 = c_add(y[1], y[3]), r3 = c_mul_mi(c_sub(y[1], y[3]));
            d[0][x] = c_add(r0, r1);
            d[1][x] = c_sub(r0, r1);
            d[2][x] = c_add(r2, r3);
            d[3][x] = c_sub(r2, r3);
        }
#pragma unroll
        for (int s = 0; s < 4; ++s) bw_tm_store(tm + 128 * pair + 32 * s, d[s]);
        bw_tm_store_wait();
    };

    // inverse outer pass of pair p's output polynomials (stored as the pair
    // level p's spectra): the last level of the second superstage, the first
    // superstage, untwist, round, centred reduction
    auto outer_inverse = [&](int pair, double (&acc_lo)[2][8], double (&acc_hi)[2][8]) {
        const int qi = ok * P + 2 * pair + oa;
        double2 v[2][8];
#pragma unroll
        for (int k2 = 0; k2 < 8; ++k2) {
            const double2 x0 = dec[bw_at(qi, oc + Q8 * k2)], x1 = dec[bw_at(qi, oc + 64 + Q8 * k2)];
            v[0][k2] = c_add(x0, x1);
            v[1][k2] = c_sub(x0, x1);
        }
#pragma unroll
        for (int col = 0; col < 2; ++col) {
            const int on1 = oc + 64 * col;
            twiddle<8, Q8, true>(v[col], tw, on1);
            dft8<true>(v[col]);
#pragma unroll
            for (int n2 = 0; n2 < 8; ++n2) {
                const double2 u = c_mul(c_conj(qtab(on1 + Q8 * n2)), v[col][n2]);
                const double rlo = rint(u.x);
                const double rhi = rint(-u.y);
                acc_lo[col][n2] = rlo - q * bw_rint_add(rlo, inv_q);
                acc_hi[col][n2] = rhi - q * bw_rint_add(rhi, inv_q);
            }
        }
    };

    // a pair's accumulators to and from tensor memory (its own columns)
    auto park_acc = [&](int pair, const double (&acc_lo)[2][8], const double (&acc_hi)[2][8]) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            double2 x[8];
#pragma unroll
            for (int n2 = 0; n2 < 8; ++n2) x[n2] = make_double2(acc_lo[h][n2], acc_hi[h][n2]);
            bw_tm_store(tm + 128 * pair + 32 * h, x);
        }
        bw_tm_store_wait();
    };
    auto unpark_acc = [&](int pair, double (&acc_lo)[2][8], double (&acc_hi)[2][8]) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            double2 x[8];
            bw_tm_load(tm + 128 * pair + 32 * h, x);
#pragma unroll
            for (int n2 = 0; n2 < 8; ++n2) {
                acc_lo[h][n2] = x[n2].x;
                acc_hi[h][n2] = x[n2].y;
            }
        }
    };

    for (long long iter = 0; iter < my_sets; ++iter) {
        const long long ct0 = (blockIdx.x + iter * gridDim.x) * K;
        double acc_lo[2][8], acc_hi[2][8];
        auto load_lut = [&](int pair) {
            const long long oct = min(ct0 + 2 * pair + ok, args.B - 1);
#pragma unroll
            for (int col = 0; col < 2; ++col)
#pragma unroll
                for (int n2 = 0; n2 < 8; ++n2) {
                    const int i = oc + 64 * col + Q8 * n2;
                    if constexpr (T64) {
                        const long long* src = args.lut64 + oct * args.lut_stride + oa * N;
                        acc_lo[col][n2] = (double)src[i];
                        acc_hi[col][n2] = (double)src[i + H];
                    } else {
                        const uint32_t* src = args.lut + oct * args.lut_stride + oa * N;
                        acc_lo[col][n2] = (double)(int32_t)src[i];
                        acc_hi[col][n2] = (double)(int32_t)src[i + H];
                    }
                }
        };
#pragma unroll 1
        for (int p = 0; p < NP; ++p) {
            load_lut(p);
            park_acc(p, acc_lo, acc_hi);
        }
        // rotation indices of every group (br_fp64_kernel's formulas)
        for (int x = tid; x < K * GM; x += BW_THREADS) {
            const int y = x / K, k = x - y * K;
            const int g = y / M, m = y - g * M;
            const long long ct = min(ct0 + k, args.B - 1);
            if constexpr (T64) {
                unsigned long long v = 0ULL;
                const unsigned long long* a = args.lwe_a64 + ct * args.lwe_n + (long long)g * args.collapse;
                for (int c = 0; c < args.collapse; ++c)
                    if ((m >> (args.collapse - 1 - c)) & 1) v += a[c];
                const int ln = __ffs(args.n_lut) - 1;
                const long long d = rne_div_pow2((long long)v, 63 - LOGN + ln);
                rot[x] = (uint16_t)((d << ln) & (2 * N - 1));
            } else {
                double v = 0.0;
                const uint32_t* a = args.lwe_a + ct * args.lwe_n + (long long)g * args.collapse;
                for (int c = 0; c < args.collapse; ++c)
                    if ((m >> (args.collapse - 1 - c)) & 1) v += (double)(int32_t)a[c];
                const double idx = rint((2.0 * N * v) / (q * args.n_lut)) * args.n_lut;
                const int ri = (int)idx % (2 * N);
                rot[x] = (uint16_t)(ri < 0 ? ri + 2 * N : ri);
            }
        }

        for (int g = 0; g < args.G; ++g) {
            // the next group's key block into L2 (all CTAs together: each its share)
            if (tid == 0 && g + 1 < args.G && args.l2_prefetch) {
                const size_t block = (size_t)2 * P * M * H * sizeof(double2);
                const size_t share = ((block / gridDim.x) + 255) & ~(size_t)255;
                const size_t off = (size_t)blockIdx.x * share;
                if (off < block) {
                    const size_t len = min(share, block - off);
                    const char* base = reinterpret_cast<const char*>(args.bsk + (size_t)(g + 1) * 2 * P * M * H);
                    prefetch_l2_bulk(base + off, (uint32_t)len);
                }
            }
#pragma unroll 1
            for (int p = 0; p < NP; ++p) {
                unpark_acc(p, acc_lo, acc_hi);
                outer_forward(acc_lo, acc_hi);
                __syncthreads();
                inner_forward(p);
                if (p + 1 < NP) __syncthreads();                     // this pair's spectra are read
            }

            // contraction: out[a] = sum_m X^{r_m} sum_bc BSK[g, a, bc, m] DEC[bc],
            // the key words of two steps (point, pattern) in flight
            {
                const double2* kb = args.bsk + (size_t)g * 2 * P * M * H + 2 * key_slot<LOGH>(warp_pos(warp * 128 + lane), L, T64);
                // key words of point s: of position bits 3 and 2, in rows slot bits 4 and 3
                auto point = [](int s) {
                    return key_order(LOGH, L, T64) == KEY_STEPS ? 64 * s : 32 * (s & 1) + 16 * (s >> 1);
                };
                const uint16_t* rg = rot + g * M * K;
                const size_t row = (size_t)M * H * 2;
                double2 kx[2][P], ky[2][P], w[K];
                auto load = [&](double2 (&kw)[2][P], const double2* p) {
#pragma unroll
                    for (int a = 0; a < 2; ++a)
#pragma unroll
                        for (int j = 0; j < P / 2; ++j)
                            ldg_pair(p + (a * (P / 2) + j) * row, kw[a][2 * j], kw[a][2 * j + 1]);
                };
                // X^r at the lane's point (root2n on the half-circle table), for
                // every ciphertext of pattern m
                auto twist = [&](int m, int e) {
                    uint32_t r2[NP];
#pragma unroll
                    for (int p = 0; p < NP; ++p) r2[p] = reinterpret_cast<const uint32_t*>(rg + m * K)[p];
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        const int idx = (int)((k & 1) ? r2[k >> 1] >> 16 : r2[k >> 1] & 0xffffu) * e;
                        const double2 x = hc[bw_root(idx & (N - 1))];
                        const int sg = (idx << (31 - LOGN)) & 0x80000000;
                        w[k] = make_double2(__hiloint2double(__double2hiint(x.x) ^ sg, __double2loint(x.x)),
                                            __hiloint2double(__double2hiint(x.y) ^ sg, __double2loint(x.y)));
                    }
                };
                load(kx, kb);
                load(ky, kb + 2 * H);
                twist(1, e0);
#pragma unroll 1
                for (int s = 0; s < 4; ++s) {
                    double2 d[NP][8], o[2][K];
#pragma unroll
                    for (int p = 0; p < NP; ++p) bw_tm_load(tm + 128 * p + 32 * s, d[p]);
#pragma unroll
                    for (int k = 0; k < K; ++k) o[0][k] = o[1][k] = make_double2(0.0, 0.0);
                    const int e = e0 + (s & 1) * N + (s >> 1) * (N / 2);
                    const int en = e0 + ((s + 1) & 1) * N + ((s + 1) >> 1) * (N / 2);
                    auto key_sum = [&](const double2 (&kw)[P], double2 (&t)[K]) {
#pragma unroll
                        for (int bc = 0; bc < P; ++bc) {
                            const double kr = kw[bc].x, ki = kw[bc].y;
#pragma unroll
                            for (int k = 0; k < K; ++k) t[k].x = fma(kr, d[k >> 1][(k & 1) * P + bc].x, t[k].x);
#pragma unroll
                            for (int k = 0; k < K; ++k) t[k].y = fma(kr, d[k >> 1][(k & 1) * P + bc].y, t[k].y);
#pragma unroll
                            for (int k = 0; k < K; ++k) t[k].x = fma(-ki, d[k >> 1][(k & 1) * P + bc].y, t[k].x);
#pragma unroll
                            for (int k = 0; k < K; ++k) t[k].y = fma(ki, d[k >> 1][(k & 1) * P + bc].x, t[k].y);
                        }
                    };
                    // one pattern, its X^r in w; w then holds the next one's
                    auto step = [&](const double2 (&kw)[2][P], int mn, int e_next) {
                        double2 wc[K];
#pragma unroll
                        for (int k = 0; k < K; ++k) wc[k] = w[k];
                        twist(mn, e_next);
#pragma unroll
                        for (int a = 0; a < 2; ++a) {
                            double2 t[K];
#pragma unroll
                            for (int k = 0; k < K; ++k) t[k] = make_double2(0.0, 0.0);
                            key_sum(kw[a], t);
#pragma unroll
                            for (int k = 0; k < K; ++k) c_mac(o[a][k], wc[k], t[k]);
                        }
                    };
                    // pattern 0 is the empty one: X^0 = 1
#pragma unroll
                    for (int a = 0; a < 2; ++a) key_sum(kx[a], o[a]);
#pragma unroll 1
                    for (int m = 0; m < M; m += 2) {
                        const bool last = m + 2 >= M;
                        const double2* nx = !last ? kb + (size_t)(m + 2) * H * 2 + point(s) : kb + point(s + 1);
                        const bool more = !last || s < 3;
                        if (m > 0) step(kx, m + 1, e);
                        if (more) load(kx, nx);
                        step(ky, last ? 1 : m + 2, last ? en : e);
                        if (more) load(ky, nx + 2 * H);
                    }
#pragma unroll
                    for (int p = 0; p < NP; ++p) {
                        // outputs in place of the point's digits: (k, a) at 2 k + a
                        double2 x[8];
#pragma unroll
                        for (int i = 0; i < 4; ++i) x[i] = o[i & 1][2 * p + (i >> 1)];
#pragma unroll
                        for (int i = 4; i < 8; ++i) x[i] = make_double2(0.0, 0.0);
                        bw_tm_store(tm + 128 * p + 32 * s, x);
                    }
                }
                bw_tm_store_wait();
            }
            // the inverse radix-16 superstage's levels at half = 8 and 4: pair
            // p's outputs in place of the spectra of level p
            {
                const double2 wa = w16t[8 + jg], wb = w16t[8 + jg + 4], wc = w16t[8 + 2 * jg];
#pragma unroll 1
                for (int p = 0; p < NP; ++p) {
                    double2 y[4][8];
#pragma unroll
                    for (int s = 0; s < 4; ++s) bw_tm_load(tm + 128 * p + 32 * s, y[s]);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const double2 s0 = c_add(y[0][i], y[1][i]), d0 = c_mul(c_sub(y[0][i], y[1][i]), wa);
                        const double2 s1 = c_add(y[2][i], y[3][i]), d1 = c_mul(c_sub(y[2][i], y[3][i]), wb);
                        const int qi = (i >> 1) * P + 2 * p + (i & 1);
                        dec[bw_at(qi, cbase)] = c_add(s0, s1);
                        dec[bw_at(qi, cbase + 2)] = c_mul(c_sub(s0, s1), wc);
                        dec[bw_at(qi, cbase + 1)] = c_add(d0, d1);
                        dec[bw_at(qi, cbase + 3)] = c_mul(c_sub(d0, d1), wc);
                    }
                }
            }
            __syncwarp();
            // inverse inner pass: both blocks of a pair's four output polynomials
#pragma unroll 1
            for (int p = 0; p < NP; ++p) {
                const int oq = (lane >> 2) & 3;
                const int qi = (oq >> 1) * P + 2 * p + (oq & 1);
                const int base = (wk + (lane >> 4)) * 128 + wh * 64 + it;
                double2 v[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = dec[bw_at(qi, base + 16 * (j >> 2) + 4 * (j & 3))];
                bw_inner_inverse(v, wh, tw1, it);
#pragma unroll
                for (int j = 0; j < 16; ++j) dec[bw_at(qi, base + 16 * (j >> 2) + 4 * (j & 3))] = v[j];
            }
            __syncthreads();
#pragma unroll 1
            for (int p = 0; p < NP; ++p) {
                outer_inverse(p, acc_lo, acc_hi);
                park_acc(p, acc_lo, acc_hi);
            }
            // no barrier: the next group's outer pass rewrites only points this
            // thread has read
        }
        __syncthreads();                                             // dec is reused below

        // epilogue: rotate by -b~ and extract, as br_fp64_kernel
        typedef typename std::conditional<T64, unsigned long long, uint32_t>::type word;
        word* acc = reinterpret_cast<word*>(smem_raw);               // [K][2][N]
        auto put_acc = [&](int pair) {
            word* dst = acc + (size_t)(2 * pair + ok) * 2 * N + oa * N;
#pragma unroll
            for (int col = 0; col < 2; ++col)
#pragma unroll
                for (int n2 = 0; n2 < 8; ++n2) {
                    const int i = oc + 64 * col + Q8 * n2;
                    if constexpr (T64) {
                        dst[i] = (word)__double2ll_rn(acc_lo[col][n2]);
                        dst[i + H] = (word)__double2ll_rn(acc_hi[col][n2]);
                    } else {
                        dst[i] = (word)(long long)acc_lo[col][n2];
                        dst[i + H] = (word)(long long)acc_hi[col][n2];
                    }
                }
        };
#pragma unroll 1
        for (int p = 0; p < NP; ++p) {
            unpark_acc(p, acc_lo, acc_hi);
            put_acc(p);
        }
        if (tid < K) {
            const long long ct = min(ct0 + tid, args.B - 1);
            if constexpr (T64) {
                const int ln = __ffs(args.n_lut) - 1;
                bexp[tid] = (int)((rne_div_pow2((long long)args.lwe_b64[ct], 63 - LOGN + ln) << ln) & (2 * N - 1));
            } else {
                const double b = (double)(int32_t)args.lwe_b[ct];
                bexp[tid] = (int)(rint((2.0 * N * b) / (q * args.n_lut)) * args.n_lut);
            }
        }
        __syncthreads();
        word *acc_out, *out_a, *out_b;
        if constexpr (T64) {
            acc_out = args.acc_out64;
            out_a = args.out_a64;
            out_b = args.out_b64;
        } else {
            acc_out = args.acc_out;
            out_a = args.out_a;
            out_b = args.out_b;
        }
        auto coef = [&](const word* p, int e) {
            e &= (2 * N - 1);
            const word v = p[e & (N - 1)];
            return (e < N) ? v : (word)(0 - v);
        };
        const int kv = (int)min((long long)K, args.B - ct0);
        if (acc_out)
            for (int x = tid; x < kv * 2 * N; x += BW_THREADS) {
                const int k = x / (2 * N), rem = x % (2 * N), a = rem / N, i = rem % N;
                acc_out[(ct0 + k) * 2 * N + rem] = coef(acc + (size_t)k * 2 * N + a * N, i + bexp[k]);
            }
        if (out_a) {
            const int nl = args.n_lut;
            for (int x = tid; x < kv * nl * N; x += BW_THREADS) {
                const int k = x / (nl * N), rem = x - k * nl * N, al = rem / N, j = rem % N;
                out_a[(ct0 + k) * nl * N + rem] = coef(acc + (size_t)k * 2 * N, al - j + bexp[k]);
            }
            for (int x = tid; x < kv * nl; x += BW_THREADS) {
                const int k = x / nl, al = x - k * nl;
                out_b[(ct0 + k) * nl + al] = coef(acc + (size_t)k * 2 * N + N, al + bexp[k]);
            }
        }
        __syncthreads();                                             // shared memory is reused by the next set
    }
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tm_base), "r"(BW_TM_COLS));
}

}  // namespace tfhe
