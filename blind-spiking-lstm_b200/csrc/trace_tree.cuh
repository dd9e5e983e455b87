// pack_lwe_to_rlwe (schemas/text_jax.py:316-345) on the 64-bit torus at N = 2048:
//   lwe <- rne(lwe / N), embedded as an RLWE (A, B);
//   for step i, k = 2^(log2 N - i) + 1: (A', B') = automorphism X -> X^k of it,
//   (A, B) += (sum_j dec_j(A') key[i][j][0], B' + sum_j dec_j(A') key[i][j][1]).
//
// One LWE per CTA of 256 threads, two CTAs per SM, whose phases (shared-memory
// passes, key loads from L2, FP64) overlap.  Against trace64_fused_kernel, which
// takes the other sizes (512 threads, one CTA per SM, every superstage behind CTA
// barriers, a key of four limbs):
//   * a 64-bit key word is three signed limbs (22, 21, 21 bits): products stay
//     below 2^43, their float64 error (at most about 60 2^-53 of that) below
//     1/16, so they round to the exact integers: six inverse transforms a step
//     instead of eight, and 3/4 of the key to read;
//   * digits come from the word's upper l log2 beta + 2 bits (the lowest one
//     sticky) in float64, exactly the integer rounding's digits;
//   * forward transforms are trees of 6-FMA butterflies without a twist
//     (br_mma.cuh), cut as there: three levels in registers, the other levels
//     and the key products by the warp that owns a block of 128 points, so four
//     CTA barriers a step are left;
//   * the transform's last level and the inverse's first run in the product's
//     registers, the inverse's outer twiddles and the untwist are one product;
//   * the words wait in tensor memory while the spectra need the registers.
// Bound by shared memory and the key loads (1184 LWEs: LSU data path 78% busy,
// FP64 45%, issue 41%).  l = 5: 296 LWEs 413 -> 284 us, 512 778 -> 485, 2048 2739 -> 1701,
// one LWE 216 -> 161, against the general kernel.  Two LWEs per CTA with shared
// key words took 549 us at 512: one CTA's phases leave the SM idle.
#pragma once

#include "br_mma.cuh"
#include "br_warp.cuh"

namespace tfhe {

constexpr int TT_LOGN = 11, TT_N = 1 << TT_LOGN, TT_H = TT_N / 2, TT_LOGH = TT_LOGN - 1;
constexpr int TT_THREADS = 256;
constexpr int TT_COL = 128;                                      // columns of the outer pass = points per block
constexpr uint32_t TT_TM_COLS = 64;
constexpr int TT_LIMBS = 3, TT_NO = 2 * TT_LIMBS;                // output spectra
constexpr int TT_NODES = 8 + 64;
// nodes, last level's factors, inverse's middle twiddles, two rows of eighths
// (odd stride), untwist of a column's points, tensor-memory address
constexpr int TT_TABLES = TT_NODES * 4 + TT_H / 2 + 112 + 17 + 8 + 1;

constexpr size_t trace_tree_smem(int l) {
    return ((size_t)(l > TT_NO ? l : TT_NO) * TT_H + TT_TABLES) * sizeof(double2);
}
static_assert(2 * (trace_tree_smem(6) + 1024) <= 228 * 1024, "two CTAs per SM");
static_assert((size_t)2 * TT_N * 8 <= (size_t)TT_NO * TT_H * 16, "the words fit in the spectra's space");

struct TraceTreeArgs {
    const unsigned long long* lwe_a;    // (R, N)
    const unsigned long long* lwe_b;    // (R)
    const double2* key;                 // [step][limb 2 + a][L][H], leaf order, times 1/H
    const double2* qt;
    const double2* tw;
    int log2_beta, steps;
    long long R;
    unsigned long long* out;            // (R, 2, N)
};

// signed limb t (22, 21, 21 bits) of a 64-bit word: w = l0 + l1 2^22 + l2 2^43
__host__ __device__ __forceinline__ long long limb3(unsigned long long w, int t) {
    const long long l0 = (long long)(w << 42) >> 42;
    const unsigned long long r = (w - (unsigned long long)l0) >> 22;             // 42 bits, modulo 2^42
    const long long l1 = (long long)(r << 43) >> 43;
    if (t == 0) return l0;
    if (t == 1) return l1;
    return (long long)((r - (unsigned long long)l1) << 22) >> 43;                // the upper 21 bits of 42
}

// exponent of the tree's node at `depth` with path bits `path`, first level first
__device__ __forceinline__ int tt_node(int depth, int path) {
    int E = TT_N >> (depth + 1);
    for (int d = 1; d <= depth; ++d)
        if ((path >> (depth - d)) & 1) E += TT_N >> (depth - d);
    return E;
}

// key polynomials (steps, L, 2, N) words -> [step][limb 2 + a][L][H]: the leaf
// of frequency j (point zeta^(4 j + 1)) at j's bits reversed, times 1/H, and the
// even points of each 64 before the odd ones (a lane takes two neighbours)
__global__ void __launch_bounds__(256) trace_key_kernel(const unsigned long long* src, int L, const double2* qt,
                                                        const double2* tw, const uint16_t* freq, double2* dst) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2* buf = reinterpret_cast<double2*>(smem_raw);
    const int poly = blockIdx.x, t = blockIdx.y;                                 // poly: (step L + level) 2 + a
    const int tid = threadIdx.x, nt = blockDim.x;
    const unsigned long long* s = src + (size_t)poly * TT_N;
    for (int i = tid; i < TT_H; i += nt) {
        const double lo = (double)limb3(s[i], t), hi = (double)limb3(s[i + TT_H], t);
        const double2 w = qt[i];
        buf[swz(i)] = make_double2(fma(w.x, lo, w.y * hi), fma(w.y, lo, -w.x * hi));
    }
    __syncthreads();
    forward_middle<TT_LOGH, 0>(buf, 1, tw, tid, nt);
    const int a = poly & 1, lvl = (poly >> 1) % L, step = (poly >> 1) / L;
    double2* d = dst + (((size_t)step * TT_NO + t * 2 + a) * L + lvl) * TT_H;
    for (int p = tid; p < TT_H; p += nt) {
        const double2 v = buf[swz(p)];
        const unsigned e = __brev((unsigned)freq[p]) >> (32 - TT_LOGH);
        d[(e & ~63u) | (e & 1) << 5 | (e & 63) >> 1] = make_double2(v.x * (1.0 / TT_H), v.y * (1.0 / TT_H));
    }
}

template <int L>
__global__ void __launch_bounds__(TT_THREADS, 2) trace_tree_kernel(const TraceTreeArgs args) {
    using Word = unsigned long long;
    constexpr int N = TT_N, H = TT_H, COL = TT_COL, NO = TT_NO;
    constexpr int PP = L > NO ? L : NO;
    using PL = Plan<TT_LOGH>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2* dec = reinterpret_cast<double2*>(smem_raw);             // [PP][H]
    Word* words = reinterpret_cast<Word*>(smem_raw);                 // [2][N], between the steps
    double2* node = dec + (size_t)PP * H;                            // 4 factors of [8] then [8][8] nodes
    double2* leaf = node + TT_NODES * 4;                             // H / 2 factors of the last level
    double2* mid = leaf + H / 2;                                     // the inverse's middle twiddles
    double2* last8 = mid + 112;                                      // 8 ones, exp(i pi k / 8)
    double2* col8 = last8 + 17;                                      // conj(zeta^(COL n))

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < TT_NODES; i += TT_THREADS) {
        const int E = i < 8 ? tt_node(3, i) : tt_node(6, i - 8);
        node[i] = root2n<TT_LOGN>(args.qt, E / 2);
        node[i + TT_NODES] = root2n<TT_LOGN>(args.qt, E / 4);
        node[i + TT_NODES * 2] = root2n<TT_LOGN>(args.qt, E / 8);
        node[i + TT_NODES * 3] = root2n<TT_LOGN>(args.qt, E / 8 + N / 4);
    }
    for (int i = tid; i < H / 2; i += TT_THREADS) leaf[i] = root2n<TT_LOGN>(args.qt, tt_node(9, i) / 2);
    if (tid < 112) mid[tid] = args.tw[PL::tw_offset(1) + tid];
    if (tid < 17) last8[tid] = tid < 9 ? make_double2(1.0, 0.0) : w16(tid - 9, true);
    if (tid < 8) col8[tid] = c_conj(args.qt[COL * tid]);

    // the words wait in tensor memory (32 columns of a warp's lanes) while the
    // spectra need the registers
    uint32_t* tm_slot = reinterpret_cast<uint32_t*>(col8 + 8);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tm_slot)),
                     "r"(TT_TM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tm_base = *tm_slot;
    const uint32_t tm = tm_base + ((uint32_t)(warp & 3) << 21) + (uint32_t)(warp >> 2) * 32;

    auto at = [](int q, int e) { return q * H + (e ^ ((e >> 3) & 7)); };
    // outer pass and words: polynomial a, coefficients c + COL n (+ H)
    const int oa = tid / COL, oc = tid % COL;
    const long long r = blockIdx.x;
    // inner passes: block `warp`, 16 lanes per polynomial
    const int t = lane & 15, pl = lane >> 4;
    const int e1 = warp * COL + t;                                   // first inner pass: + 16 j
    const int e2 = warp * COL + (t >> 1) * 16 + (t & 1);             // second: + 2 j
    const double beta = ldexp(1.0, args.log2_beta);
    const int total = L * args.log2_beta;                            // digit bits, at most 50
    const int drop = 62 - total;
    const double sc0 = ldexp(1.0, args.log2_beta - total - 2);

    Word acc[2][8];                                                  // [lower, upper half][n]
    {
        const Word* a = args.lwe_a + r * N;
        const Word b = args.lwe_b[r];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                const int i = oc + COL * n + h * H;
                const Word x = oa == 0 ? a[i == 0 ? 0 : N - i] : (i == 0 ? b : (Word)0);
                const Word ms = (Word)rne_div_pow2((long long)x, TT_LOGN);
                acc[h][n] = oa == 0 && i != 0 ? (Word)0 - ms : ms;
            }
    }

    for (int st = 0; st < args.steps; ++st) {
        // the words to shared memory, back under the automorphism: coefficient
        // i of A' is that of X^(i / k) in A, k^-1 modulo 2N
        __syncthreads();                                             // the spectra are read
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int n = 0; n < 8; ++n) words[oa * N + oc + COL * n + h * H] = acc[h][n];
        __syncthreads();
        unsigned kinv = 1u;                                          // Newton's iteration modulo 2^32
        {
            const unsigned k = (1u << (args.steps - st)) + 1u;
#pragma unroll
            for (int x = 0; x < 5; ++x) kinv *= 2u - k * kinv;
        }
        auto turned = [&](const Word* p, int i) {
            const unsigned j = ((unsigned)i * kinv) & (2 * N - 1);
            const Word v = p[j & (N - 1)];
            return j >= (unsigned)N ? (Word)0 - v : v;
        };
        double x[2][8];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                const int i = oc + COL * n + h * H;
                const Word v = turned(words, i);
                const bool rest = (v & ((1ULL << drop) - 1ULL)) != 0;
                x[h][n] = (double)(((long long)v >> drop) | (rest ? 1LL : 0LL));
                if (oa == 1) acc[h][n] += turned(words + N, i);
            }
        {
            double2 v[8];
#pragma unroll
            for (int n = 0; n < 8; ++n)
                v[n] = make_double2(__longlong_as_double((long long)acc[0][n]), __longlong_as_double((long long)acc[1][n]));
            bw_tm_store(tm, v);
            bw_tm_store_wait();
        }
        __syncthreads();

        // outer pass: gadget digits of A', the tree's first three levels; the
        // two threads of a column take the lower and the upper levels
        {
            double2 w[4];
            w[0] = make_double2(0.70710678118654752440, -0.70710678118654752440);   // zeta^(N/4)
            w[1] = make_double2(0.92387953251128675613, -0.38268343236508977173);   // zeta^(N/8)
            w[2] = make_double2(0.98078528040323044913, -0.19509032201612826785);   // zeta^(N/16)
            w[3] = make_double2(0.55557023301960222474, -0.83146961230254523708);   // zeta^(5N/16)
#pragma unroll
            for (int lvl = 0; lvl < L; ++lvl) {
                const double sc = lvl == 0 ? sc0 : beta;
                const bool mine = (lvl < (L + 1) / 2) == (oa == 0);
                if (oa == 0 && !mine) break;
                double2 v[8];
#pragma unroll
                for (int n = 0; n < 8; ++n) {
                    const double lo = bm_rint(x[0][n], sc), hi = bm_rint(x[1][n], sc);
                    x[0][n] = fma(x[0][n], sc, -lo);
                    x[1][n] = fma(x[1][n], sc, -hi);
                    v[n] = make_double2(lo, -hi);
                }
                if (mine) {
                    bm_forward8(v, w);
#pragma unroll
                    for (int n = 0; n < 8; ++n) dec[at(lvl, oc + COL * n)] = v[n];
                }
            }
        }
        __syncthreads();

        // inner passes: the warp's block of the L digit polynomials.  The 16 lanes
        // of one polynomial exchange among themselves; an odd L leaves the upper
        // half of the warp a round less
        const unsigned mask = 0xffffu << (pl * 16);
#pragma unroll 1
        for (int q = pl; q < L; q += 2) {
            double2 v[8], w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) w[i] = node[i * TT_NODES + warp];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = dec[at(q, e1 + 16 * j)];
            bm_forward8(v, w);
#pragma unroll
            for (int j = 0; j < 8; ++j) dec[at(q, e1 + 16 * j)] = v[j];
            __syncwarp(mask);
#pragma unroll
            for (int i = 0; i < 4; ++i) w[i] = node[i * TT_NODES + 8 + warp * 8 + (t >> 1)];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = dec[at(q, e2 + 2 * j)];
            bm_forward8(v, w);
#pragma unroll
            for (int j = 0; j < 8; ++j) dec[at(q, e2 + 2 * j)] = v[j];
        }
        __syncwarp();

        // key products of the block: two neighbouring points per lane, two
        // rounds; the next output's key words are on their way during one's sums
#pragma unroll 1
        for (int p = warp * COL + 2 * lane; p < (warp + 1) * COL; p += 64) {
            const double2* key = args.key + (size_t)st * NO * L * H + p - lane;
            double2 kw[L][2], d[L][2];
#pragma unroll
            for (int lvl = 0; lvl < L; ++lvl) {
                kw[lvl][0] = __ldg(key + (size_t)lvl * H);
                kw[lvl][1] = __ldg(key + (size_t)lvl * H + 32);
            }
#pragma unroll
            for (int lvl = 0; lvl < L; ++lvl) {
                d[lvl][0] = dec[at(lvl, p)];
                d[lvl][1] = dec[at(lvl, p + 1)];
                bm_bfly(d[lvl][0], d[lvl][1], leaf[p / 2]);
            }
#pragma unroll 1
            for (int o = 0; o < NO; ++o) {
                const double2* next = key + (size_t)(o + 1 < NO ? o + 1 : o) * L * H;
                double2 y0 = make_double2(0.0, 0.0), y1 = y0;
#pragma unroll
                for (int lvl = 0; lvl < L; ++lvl) {
                    c_mac(y0, d[lvl][0], kw[lvl][0]);
                    c_mac(y1, d[lvl][1], kw[lvl][1]);
                    kw[lvl][0] = __ldg(next + (size_t)lvl * H);
                    kw[lvl][1] = __ldg(next + (size_t)lvl * H + 32);
                }
                dec[at(o, p)] = c_add(y0, y1);
                dec[at(o, p + 1)] = c_sub(y0, y1);
            }
        }
        __syncwarp();

        // inverse inner passes of the output polynomials
#pragma unroll 1
        for (int o = pl; o < NO; o += 2) {
            double2 v[8], y[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) y[j] = dec[at(o, e2 + 2 * j)];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = y[bm_rev3(j)];
#pragma unroll
            for (int j = 1; j < 8; ++j) v[j] = c_mul(v[j], last8[(t & 1) * 9 + j]);
            dft8<true>(v);
#pragma unroll
            for (int j = 0; j < 8; ++j) dec[at(o, e2 + 2 * j)] = v[j];
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 8; ++j) y[j] = dec[at(o, e1 + 16 * j)];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = y[bm_rev3(j)];
            twiddle<8, 16, true>(v, mid, t);
            dft8<true>(v);
#pragma unroll
            for (int j = 0; j < 8; ++j) dec[at(o, e1 + 16 * j)] = v[j];
        }
        // conj(zeta^(c (4 j + 1))): the last superstage's twiddles and the
        // untwist's part of the column
        double2 tc[8];
        {
            tc[0] = c_conj(__ldg(args.qt + oc));
            const double2 q2 = c_mul(tc[0], tc[0]), q4 = c_mul(q2, q2), q8 = c_mul(q4, q4);
            tc[1] = c_mul(tc[0], q4);
            tc[2] = c_mul(tc[0], q8);
            tc[3] = c_mul(tc[1], q8);
            const double2 q16 = c_mul(q8, q8);
#pragma unroll
            for (int j = 0; j < 4; ++j) tc[4 + j] = c_mul(tc[j], q16);
        }
        {
            double2 v[8];
            bw_tm_load(tm, v);
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                acc[0][n] = (Word)__double_as_longlong(v[n].x);
                acc[1][n] = (Word)__double_as_longlong(v[n].y);
            }
        }
        __syncthreads();

        // last superstage, untwist, round, add
#pragma unroll 1
        for (int limb = 0; limb < TT_LIMBS; ++limb) {
            double2 v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = c_mul(dec[at(limb * 2 + oa, oc + COL * bm_rev3(j))], tc[j]);
            dft8<true>(v);
            const int sh = limb == 0 ? 0 : 22 + 21 * (limb - 1);
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                const double2 u = c_mul(col8[n], v[n]);
                acc[0][n] += (Word)__double2ll_rn(u.x) << sh;
                acc[1][n] += (Word)__double2ll_rn(-u.y) << sh;
            }
        }
    }

    Word* dst = args.out + (r * 2 + oa) * N;
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int n = 0; n < 8; ++n) dst[oc + COL * n + h * H] = acc[h][n];
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tm_base), "r"(TT_TM_COLS));
}

}  // namespace tfhe
