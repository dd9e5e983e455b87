// Batched blind rotation at N = 1024 for gadgets whose products float64 holds
// exactly, four ciphertexts per CTA of 512 threads: the key contraction on the
// FP64 matrix instruction.
//
// At n=630 (l_bs = 3, eight patterns) a group's key is 96 complex words per
// point of the spectrum and a ciphertext, and the two-per-CTA kernel spends
// two thirds of its time on it: a thread holds one point of two ciphertexts,
// reloads each key word for the next two, and has registers for one pattern's
// words at a time.  Here a warp contracts one point of four ciphertexts with
// mma.m8n8k4.f64:
//   rows    (output o, four of the patterns m): the key words of a digit pair
//           (re, im, re, im) are the four k of one row,
//   columns (ciphertext, re | im): (d.re, -d.im) and (d.im, d.re),
// so T[o][m][ct] = sum_bc BSK[g, o, bc, m] DEC[ct][bc] comes out as one complex
// number per lane, is multiplied by X^{r[ct][m]}, added over the tiles of
// four patterns in the lane and over the four rows by two shuffles.  A key word
// is loaded once for four ciphertexts and by one lane; the instruction reads
// two operands per 256 products, so the FP64 pipe is not held back by the
// register ports (a DFMA with three distinct operands takes 2.4 to 2.9 cycles
// instead of 2).
//
// Only where the rounded products are the exact integers (launcher: the
// 32-bit torus, log2 beta <= 8), so the order of sums and the transform's form
// are free and the outputs are those of br_fp64_kernel:
//   forward transform: radix-2 butterflies a + w b, 2 a - (a + w b) in 6 FMAs
//     along the tree x^H + i = (x^{H/2} - s)(x^{H/2} + s), ..., with the fold's
//     twist in the butterflies' factors (27 FP64 instructions per point
//     instead of 32, and no twist table reads); three levels per pass;
//   inverse transform: dft8 with twiddles and a final untwist, as
//     br_fp64_kernel.
// Work mapping: the outer pass (three levels, 8 points per thread in
// registers) leaves eight blocks of 64 points per polynomial; warps 2 b and
// 2 b + 1 own block b of all polynomials, so the other six levels, the
// contraction and the inverse's first six need barriers of those two warps
// only, and a group has two CTA barriers.
#pragma once

#include "br_fp64.cuh"

namespace tfhe {

constexpr int BM_THREADS = 512;
constexpr int BM_K = 4;
constexpr int BM_ROT_GROUPS = 32;                  // groups whose rotation indices are held at a time
constexpr int BM_N = 1024, BM_H = 512;
constexpr int BM_NODE = 4;                         // factors per node of a forward radix-8 pass

// shared memory of br_mma_kernel: the digit spectra of four ciphertexts, the
// half-circle roots, the inverse transform's twiddles, the forward factors of
// the 8 + 64 inner nodes, rotation indices, b~
inline size_t br_mma_smem(int L, int M) {
    return (size_t)BM_K * 2 * L * BM_H * sizeof(double2) +
           (size_t)(BM_N + Plan<9>::TW + (8 + 64) * BM_NODE) * sizeof(double2) +
           (size_t)BM_ROT_GROUPS * M * BM_K * sizeof(uint16_t) + BM_K * sizeof(int) + 16;
}

// element e of polynomial q (ciphertext k, digit bc): consecutive elements
// (outer pass, first inner pass), every eighth (second inner pass), and one
// element of the eight polynomials of a digit pair (contraction) all fall in
// distinct bank groups
template <int P>
__device__ __forceinline__ int bm_at(int k, int bc, int e) {
    return (k * P + bc) * BM_H + (e ^ ((e >> 3) & 7) ^ (k * 2 + (bc & 1)));
}

// x, y <- x + w y, x - w y
__device__ __forceinline__ void bm_bfly(double2& x, double2& y, double2 w) {
    const double2 a = x;
    x.x = fma(-w.y, y.y, fma(w.x, y.x, a.x));
    x.y = fma(w.y, y.x, fma(w.x, y.y, a.y));
    y.x = fma(2.0, a.x, -x.x);
    y.y = fma(2.0, a.y, -x.y);
}

// x, y <- x - i w y, x + i w y
__device__ __forceinline__ void bm_bfly_mi(double2& x, double2& y, double2 w) {
    const double2 a = x;
    x.x = fma(w.y, y.x, fma(w.x, y.y, a.x));
    x.y = fma(w.y, y.y, fma(-w.x, y.x, a.y));
    y.x = fma(2.0, a.x, -x.x);
    y.y = fma(2.0, a.y, -x.y);
}

// three levels of the forward tree below a node x^len = zeta^E:
// w[0..3] = zeta^(E/2), zeta^(E/4), zeta^(E/8), zeta^(E/8 + N/4); v[i]: the
// i-th eighth, then the i-th leaf (path bits, first level first)
__device__ __forceinline__ void bm_forward8(double2 (&v)[8], const double2 (&w)[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) bm_bfly(v[i], v[i + 4], w[0]);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        bm_bfly(v[i], v[i + 2], w[1]);
        bm_bfly_mi(v[4 + i], v[6 + i], w[1]);
    }
    bm_bfly(v[0], v[1], w[2]);
    bm_bfly_mi(v[2], v[3], w[2]);
    bm_bfly(v[4], v[5], w[3]);
    bm_bfly_mi(v[6], v[7], w[3]);
}

__device__ __forceinline__ constexpr int bm_rev3(int i) { return ((i & 1) << 2) | (i & 2) | (i >> 2); }

__device__ __forceinline__ void bm_mma(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(c[0]), "+d"(c[1])
        : "d"(a), "d"(b));
}

__device__ __forceinline__ void bm_pair_barrier(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }

__device__ __forceinline__ double bm_shfl(double x, int mask) { return __shfl_xor_sync(0xffffffffu, x, mask); }

// rint(x scale) for a power of two scale, |x scale| < 2^51, by adding and
// subtracting 1.5 2^52 (half to even)
__device__ __forceinline__ double bm_rint(double x, double scale) {
    constexpr double MAGIC = 6755399441055744.0;
    return __dadd_rn(fma(x, scale, MAGIC), -MAGIC);
}

__device__ __forceinline__ double2 bm_flip(double2 x, uint32_t sign) {
    return make_double2(__hiloint2double(__double2hiint(x.x) ^ (int)sign, __double2loint(x.x)),
                        __hiloint2double(__double2hiint(x.y) ^ (int)sign, __double2loint(x.y)));
}

// X^r at the four points p .. p + 3 (p a multiple of 4) for the lane's pattern
// of every tile: the points' frequencies (the position's bits reversed) differ
// by half (bit 0) and a quarter (bit 1) of the circle, so one read of the
// half-circle table gives all four, w[t][bit 1], times (-1)^r for bit 0
template <int T>
__device__ __forceinline__ void bm_twist(double2 (&w)[T][2], const int (&r)[T], const double2* hc, int p) {
    const int e = 4 * (int)(__brev((unsigned)p) >> 23) + 1;          // the point zeta^e, H = 512
#pragma unroll
    for (int t = 0; t < T; ++t) {
        const int idx = r[t] * e;
        const double2 x = bm_flip(hc[idx & (BM_N - 1)], (uint32_t)(idx << 21) & 0x80000000u);
        const double2 y = (r[t] & 1) ? c_mul_mi(x) : x;              // times (-i)^r
        w[t][0] = x;
        w[t][1] = bm_flip(y, (uint32_t)(r[t] << 30) & 0x80000000u);
    }
}

// T = key x digits of four points (2 T sums side by side: an instruction's
// result takes 28 cycles, its issue 16); reload(h) once the key words of pair
// h are consumed
template <int L, int T, class Reload>
__device__ __forceinline__ void bm_products(double (&c)[4][T][2], double2 (&ka)[T][L], double2 (&kb)[T][L],
                                            const double (&b)[4][L], Reload reload) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int s = 0; s < L; ++s)
#pragma unroll
            for (int i = 2 * h; i < 2 * h + 2; ++i)
#pragma unroll
                for (int t = 0; t < T; ++t) {
                    if (s == 0) c[i][t][0] = c[i][t][1] = 0.0;
                    const double2 k2 = h == 0 ? ka[t][s] : kb[t][s];
                    bm_mma(c[i][t], (i & 1) == 0 ? k2.x : k2.y, b[i][s]);
                }
        reload(h);
    }
}

// the four points' outputs from T: times X^r, summed over the tiles in the
// lane and over the four rows of a tile (lane bits 2 and 3); y[j] is then
// component bit 2 of point 2 j + bit 3
template <int T>
__device__ __forceinline__ void bm_sums(double (&y)[2], const double (&c)[4][T][2], const double2 (&w)[T][2],
                                        const int (&r)[T], int lane) {
    const bool b2 = lane & 4, b3 = lane & 8;
    double x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        double2 o;
#pragma unroll
        for (int t = 0; t < T; ++t) {
            const double2 f = (i & 1) ? bm_flip(w[t][i >> 1], (uint32_t)r[t] << 31) : w[t][i >> 1];
            if (t == 0) o = make_double2(f.x * c[i][t][0], f.x * c[i][t][1]);
            else o = make_double2(fma(f.x, c[i][t][0], o.x), fma(f.x, c[i][t][1], o.y));
            o.x = fma(-f.y, c[i][t][1], o.x);
            o.y = fma(f.y, c[i][t][0], o.y);
        }
        x[i] = (b2 ? o.y : o.x) + bm_shfl(b2 ? o.x : o.y, 4);
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) y[j] = (b3 ? x[2 * j + 1] : x[2 * j]) + bm_shfl(b3 ? x[2 * j] : x[2 * j + 1], 8);
}

// Double of the contraction layout: group g, warp w, pair u of its points
// (point w 32 + 2 u + sl), tile t, digit pair s, lane (row o 4 + mm, k), sl
__host__ __device__ __forceinline__ size_t bm_key_at(int L, int T, size_t g, int w, int u, int t, int s, int lane,
                                                     int sl) {
    return ((((((g * 16 + w) * 16 + u) * T + t) * L + s) * 32 + lane) * 2) + sl;
}

// native key (position order) -> contraction layout
struct BmConvArgs {
    const double2* src;
    double* dst;
    int G, M, L;
};

static __global__ void __launch_bounds__(256) bm_key_kernel(const BmConvArgs a) {
    const int T = a.M / 4, P = 2 * a.L;
    const size_t total = (size_t)a.G * 2 * P * a.M * BM_H;      // complex words
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        // i: [g][o][s][m][position][digit of the pair]
        const int dg = (int)(i & 1);
        const int p = (int)((i >> 1) % BM_H);
        size_t r = (i >> 1) / BM_H;
        const int m = (int)(r % a.M);
        r /= a.M;
        const int s = (int)(r % a.L);
        r /= a.L;
        const int o = (int)(r & 1);
        const size_t g = r >> 1;
        // position digits k0 64 + k1 8 + k2 -> leaf with every digit's bits reversed
        const int q = bm_rev3(p >> 6) * 64 + bm_rev3((p >> 3) & 7) * 8 + bm_rev3(p & 7);
        const double2 v = a.src[i];
        const int lane = (o * 4 + (m & 3)) * 4 + 2 * dg;
        const size_t at = bm_key_at(a.L, T, g, q >> 5, (q & 31) >> 1, m >> 2, s, lane, q & 1);
        a.dst[at] = v.x;
        a.dst[at + 2] = v.y;
    }
}

// the reference's key (G, 2 out, L, 2 in, M, H) at zeta^(2 j + 1), j < H ->
// contraction layout: the same points or their conjugate partners, times 1/H
// as the native key is stored (a power of two, so exact).  One block per
// (group, output, level, pattern); reads whole rows, writes 64 bytes in a row.
struct BmRefConvArgs {
    const double2* src;
    double* dst;
    int M, L;
};

static __global__ void __launch_bounds__(256) bm_ref_key_kernel(const BmRefConvArgs a) {
    __shared__ double2 row[2][BM_H];
    const int T = a.M / 4;
    const int m = blockIdx.x % a.M;
    int r = blockIdx.x / a.M;
    const int s = r % a.L;
    r /= a.L;
    const int o = r & 1;
    const size_t g = r >> 1;
    for (int i = threadIdx.x; i < 2 * BM_H; i += 256) {
        const int in = i / BM_H, j = i % BM_H;
        row[in][j] = a.src[(((((g * 2 + o) * a.L + s) * 2 + in) * a.M) + m) * BM_H + j];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 4 * (BM_H / 2); i += 256) {
        const int k = i & 3, pu = i >> 2;                            // k: digit's (re, im); pair of points
        double v[2];
#pragma unroll
        for (int sl = 0; sl < 2; ++sl) {
            const int j = (int)(__brev((unsigned)(2 * pu + sl)) >> 23), e = 4 * j + 1;
            const double2 z = e < BM_N ? row[k >> 1][2 * j] : c_conj(row[k >> 1][BM_N - 1 - 2 * j]);
            v[sl] = ((k & 1) ? z.y : z.x) * (1.0 / BM_H);
        }
        const size_t at = bm_key_at(a.L, T, g, pu >> 4, pu & 15, m >> 2, s, (o * 4 + (m & 3)) * 4 + k, 0);
        *reinterpret_cast<double2*>(a.dst + at) = make_double2(v[0], v[1]);
    }
}

// REF: the drop-in's inputs and outputs (int64 accumulators, indices given)
template <int L, int T, bool REF>
__global__ void __launch_bounds__(BM_THREADS, 1) br_mma_kernel(const BrArgs args) {
    constexpr int LOGN = 10, LOGH = 9, P = 2 * L, K = BM_K, M = 4 * T;
    constexpr int N = BM_N, H = BM_H;
    using PL = Plan<LOGH>;
    static_assert(PL::NS == 3 && PL::radix(0) == 8 && PL::radix(1) == 8 && PL::radix(2) == 8, "superstages 8.8.8");

    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2* dec = reinterpret_cast<double2*>(smem_raw);            // [K][P][H]
    double2* hc = dec + (size_t)K * P * H;                           // exp(-i pi r / N), r < N
    double2* tw = hc + N;                                            // PL::TW
    double2* node = tw + PL::TW;                                     // [8] then [8][8] nodes, 4 factors each
    uint16_t* rot = reinterpret_cast<uint16_t*>(node + (8 + 64) * BM_NODE);   // [BM_ROT_GROUPS][K][M]
    int* bexp = reinterpret_cast<int*>(rot + BM_ROT_GROUPS * K * M); // K

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long nsets = (args.B + K - 1) / K;
    const long long my_sets = blockIdx.x < nsets ? (nsets - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;

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

    // outer pass: ciphertext k, polynomial a, points c + 64 n
    const int ok = tid >> 7, oa = (tid >> 6) & 1, oc = tid & 63;
    const int blk = warp >> 1;                                       // this warp pair's block
    const int bar_id = 1 + blk;
    const int t8 = lane & 7, p4 = lane >> 3;                         // inner passes: 8 lanes per polynomial
    // contraction: B (digit k / 2 of a pair, component) of ciphertext bk
    const int bk = lane >> 3, bdig = (lane >> 1) & 1, bcomp = (lane & 1) ^ ((lane >> 2) & 1);
    const int bsign = ((lane & 1) && !((lane >> 2) & 1)) ? 0x80000000 : 0;
    // and T's (output, pattern of a tile, ciphertext) of this lane
    const int to = lane >> 4, tm = (lane >> 2) & 3, tk = lane & 3;

    const double q = ldexp(1.0, args.log2_q);
    const double inv_q = ldexp(1.0, -args.log2_q);
    const double beta = ldexp(1.0, args.log2_beta);
    const double inv_qb = ldexp(1.0, args.log2_beta - args.log2_q);
    const double* key = args.bsk_mma;

    for (long long iter = 0; iter < my_sets; ++iter) {
        const long long ct0 = (blockIdx.x + iter * gridDim.x) * K;
        double acc_lo[8], acc_hi[8];
        {
            const long long oct = min(ct0 + ok, args.B - 1);
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
        __syncthreads();

        for (int g = 0; g < args.G; ++g) {
            // the next group's key block into L2 (all CTAs together: each its share)
            if (tid == 0 && g + 1 < args.G && args.l2_prefetch) {
                const size_t block = (size_t)2 * P * M * H * sizeof(double2);
                const size_t share = ((block / gridDim.x) + 255) & ~(size_t)255;
                const size_t off = (size_t)blockIdx.x * share;
                if (off < block) {
                    const size_t len = min(share, block - off);
                    const char* base = reinterpret_cast<const char*>(key + (size_t)(g + 1) * 4 * P * M * H);
                    prefetch_l2_bulk(base + off, (uint32_t)len);
                }
            }
            // rotation indices of the next BM_ROT_GROUPS groups (br_fp64_kernel's
            // formula); the last reader of the old ones is behind a barrier
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
            {
                double2 w[4];
                w[0] = make_double2(0.70710678118654752440, -0.70710678118654752440);   // zeta^(N/4)
                w[1] = make_double2(0.92387953251128675613, -0.38268343236508977173);   // zeta^(N/8)
                w[2] = make_double2(0.98078528040323044913, -0.19509032201612826785);   // zeta^(N/16)
                w[3] = make_double2(0.55557023301960222474, -0.83146961230254523708);   // zeta^(5N/16)
#pragma unroll
                for (int lvl = 0; lvl < L; ++lvl) {
                    const double sc = lvl == 0 ? inv_qb : beta;
                    double2 v[8];
#pragma unroll
                    for (int n = 0; n < 8; ++n) {
                        const double lo = bm_rint(acc_lo[n], sc), hi = bm_rint(acc_hi[n], sc);
                        acc_lo[n] = fma(acc_lo[n], sc, -lo);
                        acc_hi[n] = fma(acc_hi[n], sc, -hi);
                        v[n] = make_double2(lo, -hi);
                    }
                    bm_forward8(v, w);
#pragma unroll
                    for (int n = 0; n < 8; ++n) dec[bm_at<P>(ok, lvl * 2 + oa, oc + 64 * n)] = v[n];
                }
            }
            __syncthreads();

            // inner passes of the pair's block: half of the polynomials each
            {
                double2 w1[4], w2[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    w1[i] = node[blk * 4 + i];
                    w2[i] = node[(8 + blk * 8 + t8) * 4 + i];
                }
#pragma unroll 1
                for (int rd = 0; rd < L; ++rd) {
                    const int q2 = (warp & 1) * 4 * L + rd * 4 + p4;   // of K P = 8 L polynomials
                    const int k = q2 / P, bc = q2 % P;
                    double2 v[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) v[j] = dec[bm_at<P>(k, bc, blk * 64 + t8 + 8 * j)];
                    bm_forward8(v, w1);
#pragma unroll
                    for (int j = 0; j < 8; ++j) dec[bm_at<P>(k, bc, blk * 64 + t8 + 8 * j)] = v[j];
                    __syncwarp();
#pragma unroll
                    for (int j = 0; j < 8; ++j) v[j] = dec[bm_at<P>(k, bc, blk * 64 + 8 * t8 + j)];
                    bm_forward8(v, w2);
#pragma unroll
                    for (int j = 0; j < 8; ++j) dec[bm_at<P>(k, bc, blk * 64 + 8 * t8 + j)] = v[j];
                }
            }
            bm_pair_barrier(bar_id);

            // contraction of this warp's 32 points, two at a time, the key
            // words of two pairs of points in flight
            {
                const double2* kp = reinterpret_cast<const double2*>(key + bm_key_at(L, T, g, warp, 0, 0, 0, lane, 0));
                constexpr int STEP = T * L * 32;                     // double2 per pair of points
                int rr[T];
                const uint16_t* rg = rot + (g % BM_ROT_GROUPS) * K * M + tk * M + tm;
#pragma unroll
                for (int t = 0; t < T; ++t) rr[t] = rg[4 * t];
                double2 ka[T][L], kb[T][L];
                auto load = [&](double2 (&kw)[T][L], int u) {
#pragma unroll
                    for (int t = 0; t < T; ++t)
#pragma unroll
                        for (int s = 0; s < L; ++s) kw[t][s] = __ldg(kp + (size_t)u * STEP + (t * L + s) * 32);
                };
                const double* bbase = reinterpret_cast<const double*>(dec + (bk * P + bdig) * H) + bcomp;
                const int bx = bk * 2 + bdig;                        // bm_at's exclusive-or of this lane's digits
                const int p0 = warp * 32;
                load(ka, 0);
                load(kb, 1);
#pragma unroll 1
                for (int u = 0; u < 16; u += 2) {
                    double c[4][T][2], b[4][L], y[2];
                    double2 w[T][2];
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int s = 0; s < L; ++s) {
                            const int p = p0 + 2 * u + i;
                            const double x = bbase[(size_t)(2 * s * H + (p ^ ((p >> 3) & 7) ^ bx)) * 2];
                            b[i][s] = __hiloint2double(__double2hiint(x) ^ bsign, __double2loint(x));
                        }
                    bm_products<L, T>(c, ka, kb, b, [&](int h) {
                        if (u < 14) {
                            if (h == 0) load(ka, u + 2);
                            else load(kb, u + 3);
                        }
                    });
                    bm_twist<T>(w, rr, hc, p0 + 2 * u);
                    bm_sums<T>(y, c, w, rr, lane);
#pragma unroll
                    for (int j = 0; j < 2; ++j)
                        reinterpret_cast<double*>(dec + bm_at<P>(tk, to, p0 + 2 * (u + j) + ((lane >> 3) & 1)))[(lane >> 2) & 1] = y[j];
                }
            }
            bm_pair_barrier(bar_id);

            // inverse inner passes of the block's output polynomials, four per warp
            {
                const int q2 = (warp & 1) * 4 + p4;
                const int k = q2 >> 1, bc = q2 & 1;
                double2 v[8], x[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) x[j] = dec[bm_at<P>(k, bc, blk * 64 + 8 * t8 + j)];
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = x[bm_rev3(j)];
                dft8<true>(v);
#pragma unroll
                for (int j = 0; j < 8; ++j) dec[bm_at<P>(k, bc, blk * 64 + 8 * t8 + j)] = v[j];
                __syncwarp();
#pragma unroll
                for (int j = 0; j < 8; ++j) x[j] = dec[bm_at<P>(k, bc, blk * 64 + t8 + 8 * j)];
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = x[bm_rev3(j)];
                twiddle<8, 8, true>(v, tw + PL::tw_offset(1), t8);
                dft8<true>(v);
#pragma unroll
                for (int j = 0; j < 8; ++j) dec[bm_at<P>(k, bc, blk * 64 + t8 + 8 * j)] = v[j];
            }
            __syncthreads();

            // last superstage, untwist, round, centred reduction
            {
                double2 v[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = dec[bm_at<P>(ok, oa, oc + 64 * bm_rev3(j))];
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
            }
            // no barrier: the next outer pass rewrites points of output
            // polynomials that this thread has read, and digit polynomials whose
            // last readers are behind the barrier above
        }
        __syncthreads();                                             // dec is reused below

        if constexpr (REF) {
            if (ct0 + ok < args.B) {
                int64_t* dst = args.out_i64 + (ct0 + ok) * 2 * N + oa * N;
#pragma unroll
                for (int n = 0; n < 8; ++n) {
                    dst[oc + 64 * n] = __double2ll_rn(acc_lo[n]);
                    dst[oc + 64 * n + H] = __double2ll_rn(acc_hi[n]);
                }
            }
            continue;
        }
        // epilogue: rotate by -b~ and extract, as br_fp64_kernel
        uint32_t* acc = reinterpret_cast<uint32_t*>(smem_raw);       // [K][2][N]
        {
            uint32_t* dst = acc + (size_t)ok * 2 * N + oa * N;
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                dst[oc + 64 * n] = (uint32_t)(long long)acc_lo[n];
                dst[oc + 64 * n + H] = (uint32_t)(long long)acc_hi[n];
            }
        }
        if (tid < K) {
            const double b = (double)(int32_t)args.lwe_b[min(ct0 + tid, args.B - 1)];
            bexp[tid] = (int)(rint((2.0 * N * b) / (q * args.n_lut)) * args.n_lut);
        }
        __syncthreads();
        const int kv = (int)min((long long)K, args.B - ct0);
        if (args.acc_out)
            for (int x = tid; x < kv * 2 * N; x += BM_THREADS) {
                const int k = x / (2 * N), rem = x % (2 * N), a = rem / N, i = rem % N;
                args.acc_out[(ct0 + k) * 2 * N + rem] = ncoef<LOGN>(acc + (size_t)k * 2 * N + a * N, i + bexp[k]);
            }
        if (args.out_a) {
            const int nl = args.n_lut;
            for (int x = tid; x < kv * nl * N; x += BM_THREADS) {
                const int k = x / (nl * N), rem = x - k * nl * N, al = rem / N, j = rem % N;
                args.out_a[(ct0 + k) * nl * N + rem] = ncoef<LOGN>(acc + (size_t)k * 2 * N, al - j + bexp[k]);
            }
            for (int x = tid; x < kv * nl; x += BM_THREADS) {
                const int k = x / nl, al = x - k * nl;
                args.out_b[(ct0 + k) * nl + al] = ncoef<LOGN>(acc + (size_t)k * 2 * N + N, al + bexp[k]);
            }
        }
        __syncthreads();                                             // shared memory is reused by the next set
    }
}

}  // namespace tfhe
