// Complex128 GEMMs of the FP64 factorisation on the 5th-generation tensor cores, by
// splitting into integer digits (the error-free transformation of Ozaki, Ogita, Oishi and
// Rump, Numer. Algorithms 59, 2012): GB300's FP64 pipe does two multiply-adds per SM and
// clock, its FP16 tensor cores about four thousand.
//
// Scaling.  C = A B with inner index k: row k of B is divided by 2^rho_k, its largest
// exponent (taken over the two matrices, G and H or L and U, that meet the same A), column
// k of A is multiplied by it, then every row i of A and column j of B by its own power of
// two, so that all entries lie in (-1, 1).  The powers are exact; rho keeps an unknown of
// another magnitude from losing its digits (the columns of L grow as the fourth power of
// the radial order, the rows of G fall as fast).
//
// Digits.  An entry is rounded to 63 bits and written as nine digits in [-64, 64] of base
// 128, exact in FP16:  x = 2 sum_i x_i 128^-(i+1).  The product keeps the 45 digit pairs with
// i + i' = d <= 8:  4 sum_d 128^-(d+2) (sum over pairs and k of x_i y_i').  A real or imaginary
// part takes two real products per k, so the inner sum of one d is a sum of 2 (d + 1) K
// products of at most 2^12: an integer of at most 2^24 for (d + 1) K <= 2048, and exact in the
// MMA's FP32 accumulators.  Longer inner dimensions are cut: at 224 for d = 8-6, 336 for 5-3 and
// 672 for 2-0.  The nine sums are put together as integers and rounded to FP64 once.
//
// What is lost, in units of the powers of two that scale row and column: 2^-62 per real product
// by rounding the entries, 1.01 x 2^-60 by the pairs left out (d >= 9), two such products per
// k.  The powers are below twice the largest components, so a real or imaginary part of C is
// off by at most 10.1 K 2^-60 of (largest of A's row) x (largest of B's column), after the
// scaling by rho, and one rounding.  That is a bound by rows and columns.  An entry of C whose
// own sum |a||b| is far below that product of maxima, which rho cannot repair when the grading
// is not one of rows, columns and inner index (entries that fall off from the diagonal, weakly
// coupled unknowns), has less relative accuracy than FP64 multiply-adds would give it.
// Measured on forced solves, against solutions refined with residuals in quadruple precision,
// largest of three frequencies, FP64 multiply-adds and digits: whole solution of the magnetic
// shell (blocks of 90 to 300) 2.4e-12 to 6.9e-11 and 4.9e-12 to 8.1e-11, every section alike;
// of the hydrodynamic shell 2.9e-13 and 2.1e-13 (S = 160), 4.9e-12 and 1.9e-12 (240); every
// degree down to 1e-20 of the largest as before or better.  Single coefficients above 1e-6, 1e-8
// and 1e-12 of the largest: 5e-10 and 8e-10, 4e-8, 8e-5 of themselves (160), 1e-9 to 7e-9 and
// 2e-8, 1.5e-6, 3.5e-3 (240): up to 1.5e-14 of the largest, below the error of the whole.
// (Scales of their own for every 32 k keep those too, but each 32 k's sum then has to be rounded
// and added in FP64: four shifts of the 72k-unknown shell 94 -> 134 ms.)
//
// Data flow.  k_oz_rho finds rho; k_oz_split_a and k_oz_split_b write the digit planes in
// the order the MMA reads them (8 x 16-byte core matrices, K-major, no swizzle), nine slices
// of a 16-wide step of K one after another, so a step is one contiguous bulk copy.
// k_oz_gemm computes a 128 x 64 tile: the tensor memory holds the accumulators of three
// values of d (Re and Im: 384 columns), so the tile takes three passes over K, d = 8-6 with
// nine slices, 5-3 with six, 2-0 with three; one thread issues tcgen05.mma (kind::f16), one
// the bulk copies into a two-stage ring (108 KB per stage), and sixteen warps move the
// sums into 64-bit integers between the passes.
// What bounds it: 180 MMAs per step of K, 84 cycles each with everything that a tile of S = 240
// takes, of which the tensor pipe is busy for 32 (38% of the active cycles; DRAM 7%, L2 10%, the
// L1 and shared-memory unit 57%).  An MMA of 128 x 64 x 16 reads 6 KB of shared memory, 48 cycles
// at 128 bytes a cycle; the rest is the passes' starts and drains, during which no MMA runs.
#include "kore_internal.cuh"
#include "kore_tma.cuh"
#include <algorithm>
#include <cstring>
#include <vector>

namespace {

constexpr int kOzSlices = 9, kOzBits = 7;
constexpr int kOzM = 128, kOzN = 64, kOzK = 16;
constexpr int kOzSliceA = 2 * kOzM * kOzK * 2;     // bytes of one slice of a step: Re, Im
constexpr int kOzSliceB = 2 * kOzN * kOzK * 2;
constexpr int kOzStepA = kOzSlices * kOzSliceA, kOzStepB = kOzSlices * kOzSliceB;
constexpr int kOzStages = 2;
constexpr int kOzStage = kOzStepA + kOzStepB;      // 108 KB
constexpr int kOzEpiWarps = 16;
constexpr int kOzThreads = 32 * (kOzEpiWarps + 2); // + the copying and the MMA warp
constexpr size_t kOzSmem = (size_t)kOzStages * kOzStage + 128 + 128;
constexpr int kOzNone = -100000;                   // exponent of an all-zero row
constexpr int kOzBad = 100000;                     // exponent of a row with an infinity or NaN
// rho of a zero row of B: the column of A that meets it takes no part in the scale of A's rows.
// (Left as it stands it decides that scale wherever its entries are the largest, and the others
// lose their digits: boundary rows have no couplings, so L has zero rows, and solutions that
// fall off with the degree had blocks of 1e-12 of the largest off by 1e-6 of themselves, 1e-12
// with it.)
constexpr int kOzUnused = -4096;

// A pass g sums the pairs of d = 8 - 3 g, 7 - 3 g, 6 - 3 g.  Steps of K that one pass may take:
// two real products of 9 - 3 g pairs at most per k, each at most 64^2, stay within 2^24.
constexpr int kOzPasses = 3;
__host__ __device__ constexpr int oz_max_steps(int g) { return (1 << 24) / (2 * (kOzSlices - 3 * g) * kOzK * 4096); }
static_assert(oz_max_steps(0) == 14 && oz_max_steps(1) == 21 && oz_max_steps(2) == 42, "exact FP32 sums");
// `steps` of K are cut into this many pieces for pass g, piece p being [p steps / n, (p + 1) steps / n).
// The pieces of the last pass are segments: each is a product of its own, rounded and added to
// C, whose passes 0 and 1 are cut further but summed as integers.
__host__ __device__ constexpr int oz_pieces(int steps, int g) { return (steps + oz_max_steps(g) - 1) / oz_max_steps(g); }
constexpr int kOzPlainSteps = oz_max_steps(0);   // up to this many nothing is cut

int oz_mt(int S) { return (S + kOzM - 1) / kOzM; }
int oz_nt(int S) { return (S + kOzN - 1) / kOzN; }
__host__ __device__ inline int oz_steps(int S) { return (S + kOzK - 1) / kOzK; }
// planes of S rows (columns) and an inner dimension K
int64_t oz_bytes_a(int S, int K) { return (int64_t)oz_mt(S) * oz_steps(K) * kOzStepA; }
int64_t oz_bytes_b(int S, int K) { return (int64_t)oz_nt(S) * oz_steps(K) * kOzStepB; }

// The scaling of an inner dimension: rows of X0 and X1 (X1 may be null).
struct OzPair {
    const double2 *X0, *X1;
};
// A matrix to split, and the pair whose rho scales it.
struct OzOperand {
    const double2 *X;
    int pair;
};
// C = beta C + alpha (A1 B1 [+ A2 B2]): indices of split operands (a2 < 0: one product).
struct OzJob {
    int a1, b1, a2, b2;
    double2 *C;
    int negate, beta;
};

// The transform E of a group of columns [g0, g1) of the Gauss-Jordan work matrices and the
// columns it is applied to: t <- t (zero in the group's pivot rows) + E t[pivot rows], for
// block z = first + i (i: the batch's), shift z / nodd of the factor window, odd index
// z % nodd.  Before the first group's update the columns are the diagonal block's.
struct OzGroup {
    double2 *T;
    const double2 *D;
    const int *piv, *used;
    int64_t t_stride, t_block, f_stride, p_stride;
    int nodd, stride, S, g0, g1, first;
    __device__ double2 *work(int i) const {
        const int z = first + i, sh = z / nodd, o = z - sh * nodd;
        return T + sh * t_stride + o * t_block;
    }
    __device__ const double2 *source(int i) const {
        if (g0 != 0) return work(i);
        const int z = first + i, sh = z / nodd, o = z - sh * nodd;
        return D + sh * f_stride + (2 * o + 1) * stride * (int64_t)S * S;
    }
    __device__ int64_t rows(int i) const {   // offset of the block's piv and used
        const int z = first + i, sh = z / nodd, o = z - sh * nodd;
        return sh * p_stride + (int64_t)o * S;
    }
    __device__ int column(int t) const { return t < g0 ? t : t + g1 - g0; }   // t-th column outside the group
};

// exponent e with |v| < 2^e of a finite nonzero double, from its bits (all subnormals: -1022)
__device__ __forceinline__ int exp_of(double2 v) {
    const int a = (__double2hiint(v.x) >> 20) & 0x7ff, b = (__double2hiint(v.y) >> 20) & 0x7ff;
    const int m = max(a, b);
    if (m == 0) return ((__double_as_longlong(v.x) | __double_as_longlong(v.y)) << 1) == 0 ? kOzNone : -1022;
    return m == 0x7ff ? kOzBad : m - 1022;
}

// rho of a row of B with largest exponent e
__device__ __forceinline__ int rho_of(int e) { return e == kOzNone ? kOzUnused : e == kOzBad ? 0 : e; }

// rho[pair][k] = largest exponent in row k of the pair's matrices.  CTA = 32 rows, warps
// over the columns.
__global__ void __launch_bounds__(256) k_oz_rho(const OzPair *__restrict__ pairs, int S, int *__restrict__ rho) {
    __shared__ int sm[8][32];
    const OzPair p = pairs[blockIdx.y];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, r = blockIdx.x * 32 + lane;
    int e = kOzNone;
    if (r < S)
        for (int c = w; c < S; c += 8) {
            e = max(e, exp_of(p.X0[r + (int64_t)c * S]));
            if (p.X1) e = max(e, exp_of(p.X1[r + (int64_t)c * S]));
        }
    sm[w][lane] = e;
    __syncthreads();
    if (w == 0 && r < S) {
#pragma unroll
        for (int q = 1; q < 8; ++q) e = max(e, sm[q][lane]);
        rho[(int64_t)blockIdx.y * S + r] = rho_of(e);
    }
}

// v 2^(62 - e) rounded to an integer (|v| < 2^e)
__device__ __forceinline__ long long fixed63(double v, int e) {
    const long long b = __double_as_longlong(v);
    const int ex = (int)(b >> 52) & 0x7ff;
    if (ex == 0x7ff) return 0;
    const long long m = (b & 0xfffffffffffffll) | (ex ? 1ll << 52 : 0);
    const int sh = max(ex, 1) - 1075 + 62 - e;
    long long x;
    if (sh >= 0) x = sh <= 10 ? m << sh : 0;   // sh <= 9 by |v| < 2^e, 10 for a subnormal
    else x = sh > -55 ? (m + (1ll << (-sh - 1))) >> -sh : 0;
    return b < 0 ? -x : x;
}

// The nine digits of eight fixed-point numbers x, packed as the eight FP16 values (16 bytes)
// of each slice.
__device__ __forceinline__ void put_digits(long long (&x)[8], unsigned char *out, int64_t stride) {
#pragma unroll
    for (int s = kOzSlices - 1; s >= 0; --s) {
        uint32_t h[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            int d;
            if (s > 0) {
                d = (((int)x[u] + 64) & 127) - 64;
                x[u] = (x[u] - d) >> kOzBits;
            } else d = (int)x[u];
            h[u] = (uint32_t)(0x6600 + d);   // FP16 bits of 1536 + d
        }
        uint4 v;
        uint32_t *p = &v.x;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t w = h[2 * u] | (h[2 * u + 1] << 16);
            uint32_t r;
            asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(w), "r"(0x66006600u));   // exact
            p[u] = r;
        }
        *reinterpret_cast<uint4 *>(out + s * stride) = v;
    }
}

// Planes and row exponents of an A operand: 32 rows per CTA (grid x), operand = blockIdx.y.
// The planes' order: [row tile of 128][step of K][slice][Re, Im][8 rows][half step][row][8 k].
__device__ __forceinline__ void split_a(const double2 *__restrict__ X, int S, int K, const int *__restrict__ rho,
                                        unsigned char *__restrict__ planes, int64_t bytes, int *__restrict__ exps) {
    __shared__ int sm[8][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, r = blockIdx.x * 32 + lane;
    int e = kOzNone;
    if (r < S)
        for (int k = w; k < K; k += 8) {
            const int x = exp_of(X[r + (int64_t)k * S]);
            e = max(e, (x == kOzNone || x == kOzBad) ? x : x + rho[k]);
        }
    sm[w][lane] = e;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 8; ++q) e = max(e, sm[q][lane]);
    if (w == 0 && r < S) exps[(int64_t)blockIdx.y * S + r] = e;
    if (r >= S) return;
    const int steps = oz_steps(K);
    unsigned char *base = planes + (int64_t)blockIdx.y * bytes + (int64_t)(r / kOzM) * steps * kOzStepA +
                          ((r % kOzM) / 8) * 256 + (r % 8) * 16;
    for (int kg = w; kg < 2 * steps; kg += 8) {
        long long re[8], im[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int k = kg * 8 + u;
            const double2 v = k < K ? X[r + (int64_t)k * S] : mk(0.0, 0.0);
            const int ek = k < K ? e - rho[k] : 0;
            re[u] = fixed63(v.x, ek);
            im[u] = fixed63(v.y, ek);
        }
        unsigned char *o = base + (int64_t)(kg >> 1) * kOzStepA + (kg & 1) * 128;
        put_digits(re, o, kOzSliceA);
        put_digits(im, o + kOzSliceA / 2, kOzSliceA);
    }
}

__global__ void __launch_bounds__(256) k_oz_split_a(const OzOperand *__restrict__ ops, int S,
                                                    const int *__restrict__ rho, unsigned char *__restrict__ planes,
                                                    int64_t bytes, int *__restrict__ exps) {
    const OzOperand op = ops[blockIdx.y];
    split_a(op.X, S, S, rho + (int64_t)op.pair * S, planes, bytes, exps);
}
__global__ void __launch_bounds__(256) k_oz_group_a(const OzGroup q, const int *__restrict__ rho,
                                                    unsigned char *__restrict__ planes, int64_t bytes,
                                                    int *__restrict__ exps) {
    const int W = q.g1 - q.g0;
    split_a(q.work(blockIdx.y) + (int64_t)q.g0 * q.S, q.S, W, rho + (int64_t)blockIdx.y * W, planes, bytes, exps);
}

// Planes and column exponents of a B operand: 8 columns per CTA (grid x), a warp's lanes
// over the columns; the planes' order as above with columns in the place of rows and tiles
// of 64.
// Column c of n, entry k of K: X[row(k) + ld c], row(k) = k or the pivot row of k.
__device__ __forceinline__ void split_b(const double2 *__restrict__ X, const int *__restrict__ piv, int c, int n, int K,
                                        const int *__restrict__ rho, unsigned char *__restrict__ planes, int64_t bytes,
                                        int *__restrict__ exps) {
    __shared__ int sm[32][8];
    const int c8 = threadIdx.x & 7, t = threadIdx.x >> 3;   // 8 columns x 32
    auto at = [&](int k) { return X[piv ? piv[k] : k]; };
    int e = kOzNone;
    if (c < n)
        for (int k = t; k < K; k += 32) {
            const int x = exp_of(at(k));
            e = max(e, (x == kOzNone || x == kOzBad) ? x : x - rho[k]);
        }
    sm[t][c8] = e;
    __syncthreads();
#pragma unroll 8
    for (int q = 0; q < 32; ++q) e = max(e, sm[q][c8]);
    if (t == 0 && c < n) exps[(int64_t)blockIdx.y * n + c] = e;
    if (c >= n) return;
    const int steps = oz_steps(K);
    unsigned char *base = planes + (int64_t)blockIdx.y * bytes + (int64_t)(c / kOzN) * steps * kOzStepB +
                          ((c % kOzN) / 8) * 256 + (c % 8) * 16;
    for (int kg = t; kg < 2 * steps; kg += 32) {
        long long re[8], im[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int k = kg * 8 + u;
            const double2 v = k < K ? at(k) : mk(0.0, 0.0);
            const int ek = k < K ? e + rho[k] : 0;
            re[u] = fixed63(v.x, ek);
            im[u] = fixed63(v.y, ek);
        }
        unsigned char *o = base + (int64_t)(kg >> 1) * kOzStepB + (kg & 1) * 128;
        put_digits(re, o, kOzSliceB);
        put_digits(im, o + kOzSliceB / 2, kOzSliceB);
    }
}
__global__ void __launch_bounds__(256) k_oz_split_b(const OzOperand *__restrict__ ops, int S,
                                                    const int *__restrict__ rho, unsigned char *__restrict__ planes,
                                                    int64_t bytes, int *__restrict__ exps) {
    const OzOperand op = ops[blockIdx.y];
    const int c = blockIdx.x * 8 + (threadIdx.x & 7);
    split_b(op.X + (int64_t)c * S, nullptr, c, S, S, rho + (int64_t)op.pair * S, planes, bytes, exps);
}
__global__ void __launch_bounds__(256) k_oz_group_b(const OzGroup q, const int *__restrict__ rho,
                                                    unsigned char *__restrict__ planes, int64_t bytes,
                                                    int *__restrict__ exps) {
    const int W = q.g1 - q.g0, c = blockIdx.x * 8 + (threadIdx.x & 7);
    split_b(q.source(blockIdx.y) + (int64_t)q.column(c) * q.S, q.piv + q.rows(blockIdx.y) + q.g0, c, q.S - W, W,
            rho + (int64_t)blockIdx.y * W, planes, bytes, exps);
}
// rho of a group: the largest exponent of each of its pivot rows outside the group.  One CTA
// per block, a warp per pivot row.
__global__ void __launch_bounds__(512) k_oz_group_rho(const OzGroup q, int *__restrict__ rho) {
    const int W = q.g1 - q.g0, n = q.S - W, lane = threadIdx.x & 31;
    const double2 *X = q.source(blockIdx.x);
    const int *piv = q.piv + q.rows(blockIdx.x) + q.g0;
    for (int k = threadIdx.x >> 5; k < W; k += 16) {
        int e = kOzNone;
        for (int t = lane; t < n; t += 32) e = max(e, exp_of(X[piv[k] + (int64_t)q.column(t) * q.S]));
        e = __reduce_max_sync(0xffffffffu, e);
        if (lane == 0) rho[(int64_t)blockIdx.x * W + k] = rho_of(e);
    }
}

// ----------------------------------------------------------------------------- tcgen05 PTX
__device__ __forceinline__ void oz_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void oz_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void oz_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void oz_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void oz_ld8(uint32_t taddr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void oz_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// bulk copy of `bytes` (a multiple of 16) contiguous bytes global -> shared, completing on bar
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
// Shared-memory descriptor of a K-major operand of 8 x 16-byte core matrices without
// swizzle: leading byte offset (the next core matrix along K) 128, stride byte offset (the
// next 8 rows) 256, version 1.
__device__ __forceinline__ uint64_t core_desc(uint32_t saddr) {
    return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(256 >> 4) << 32) |
           ((uint64_t)1 << 46);
}
// Instruction descriptor of kind::f16: D F32 (bits 4-5 = 1), A and B F16 (0), A negated
// (bit 13), N >> 3 at bits 17-22, M >> 4 at bits 24-28.
__host__ __device__ constexpr uint32_t f16_idesc(int negate_a) {
    return (1u << 4) | ((uint32_t)negate_a << 13) | ((uint32_t)(kOzN >> 3) << 17) | ((uint32_t)(kOzM >> 4) << 24);
}

struct OzParams {
    const OzJob *jobs;
    const unsigned char *pa, *pb;     // split operands
    const int *ea, *eb;               // their exponents, S each
    int64_t bytes_a, bytes_b;         // of one split operand
    int S, nt, steps;                 // rows (and leading dimension) of C, column tiles, steps of K
    int *err;
    OzGroup group;                    // group update: block blockIdx.y instead of a job
};

// (h 2^42 + g) 2^(e - 68) rounded to FP64
__device__ __forceinline__ double from_digits(long long h, long long g, int e) {
    const __int128 v = ((__int128)h << 42) + g;
    const bool neg = v < 0;
    unsigned __int128 u = neg ? -(unsigned __int128)v : (unsigned __int128)v;
    const unsigned long long hi = (unsigned long long)(u >> 64), lo = (unsigned long long)u;
    if ((hi | lo) == 0) return 0.0;
    const int lz = hi ? __clzll((long long)hi) : 64 + __clzll((long long)lo);
    u <<= lz;
    const unsigned long long m = (unsigned long long)(u >> 64);           // v = m 2^(64 - lz)
    const unsigned long long m53 = (m >> 11) + ((m >> 10) & 1);           // = m53 2^(75 - lz)
    const int q = 75 - lz + e - 68, be = q + 1075;
    double r;
    if (be >= 1 && be < 2046)   // m53 = 2^53 carries into the exponent
        r = __longlong_as_double((long long)(((unsigned long long)be << 52) + (m53 - (1ull << 52))));
    else r = ldexp((double)m53, q);
    return neg ? -r : r;
}

// One 128 x 64 tile (blockIdx.x) of job (of the group update: block) blockIdx.y.  CUT: more
// than kOzPlainSteps steps.  (The 64 registers of a thread's integer sums leave too few for the
// rest: of the 96 that eighteen warps have, 516 bytes a thread spill with CUT, 312 without and
// 200 in the group update.)
template <bool GROUP, bool CUT>
__global__ void __launch_bounds__(kOzThreads, 1) k_oz_gemm(const OzParams P) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + kOzStages * kOzStage);
    uint64_t *empty = full + kOzStages;
    uint64_t *accum = empty + kOzStages;     // a pass's sums are complete
    uint64_t *drained = accum + 1;           // and have been read
    uint32_t *holder = reinterpret_cast<uint32_t *>(drained + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int S = P.S, steps = P.steps;
    OzJob job;
    if (GROUP) {
        job.a1 = job.b1 = blockIdx.y;
        job.a2 = job.b2 = -1;
        job.C = P.group.work(blockIdx.y);
        job.negate = 0;
        job.beta = 1;
    } else job = P.jobs[blockIdx.y];
    const int ncols = GROUP ? S - (P.group.g1 - P.group.g0) : S;
    const int mt = blockIdx.x / P.nt, nt = blockIdx.x - mt * P.nt;
    const int parts = CUT ? oz_pieces(steps, 2) : 1;   // segments of a product
    const int nseg = (job.a2 >= 0 ? 2 : 1) * parts;
    if (tid == 0) {
        for (int s = 0; s < kOzStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(accum, 1);
        mbar_init(drained, kOzEpiWarps);
        mbar_fence_init();
    }
    if (warp == kOzEpiWarps + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(holder))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    oz_fence_before();
    __syncthreads();
    oz_fence_after();
    const uint32_t tmem = *holder;

    if (warp == kOzEpiWarps) {
        if (lane == 0) {
            uint32_t it = 0;
            for (int sg = 0; sg < nseg; ++sg) {
                const int prod = sg / parts, part = sg - prod * parts;
                const int k0 = part * steps / parts, k1 = (part + 1) * steps / parts;
                const unsigned char *pa = P.pa + (prod ? job.a2 : job.a1) * P.bytes_a + (int64_t)mt * steps * kOzStepA;
                const unsigned char *pb = P.pb + (prod ? job.b2 : job.b1) * P.bytes_b + (int64_t)nt * steps * kOzStepB;
                for (int g = 0; g < kOzPasses; ++g) {
                    const uint32_t ns = kOzSlices - 3 * g;
                    for (int k = k0; k < k1; ++k, ++it) {   // the pieces of a pass follow one another
                        const int s = it % kOzStages;
                        if (!mbar_wait(&empty[s], ((it / kOzStages) & 1u) ^ 1u)) atomicCAS(P.err, 0, KORE_DEVERR_FLAG);
                        mbar_arrive_expect_tx(&full[s], ns * (kOzSliceA + kOzSliceB));
                        unsigned char *sa = smem + (size_t)s * kOzStage;
                        bulk_load(sa, pa + (int64_t)k * kOzStepA, ns * kOzSliceA, &full[s]);
                        bulk_load(sa + kOzStepA, pb + (int64_t)k * kOzStepB, ns * kOzSliceB, &full[s]);
                    }
                }
            }
            // every copy has landed before the CTA may exit (normally already read)
            for (uint32_t i = it > kOzStages ? it - kOzStages : 0; i < it; ++i)
                if (!mbar_wait(&full[i % kOzStages], (i / kOzStages) & 1u)) atomicCAS(P.err, 0, KORE_DEVERR_FLAG);
        }
        __syncwarp();
    } else if (warp == kOzEpiWarps + 1) {
        if (lane == 0) {
            uint32_t it = 0, pass = 0;
            // the passes of all segments, each in its pieces
            for (int g3 = 0; g3 < nseg * kOzPasses; ++g3) {
                const int sg = g3 / kOzPasses, g = g3 - sg * kOzPasses, part = sg % parts;
                const int s0 = part * steps / parts, n = (part + 1) * steps / parts - s0;
                const int np = CUT ? oz_pieces(n, g) : 1;
                for (int p = 0; p < np; ++p, ++pass) {
                    const int k0 = s0 + p * n / np, k1 = s0 + (p + 1) * n / np;
                    if (pass > 0 && !mbar_wait(drained, (pass - 1) & 1u)) atomicCAS(P.err, 0, KORE_DEVERR_FLAG);
                    oz_fence_after();
                    for (int k = k0; k < k1; ++k, ++it) {
                        const int s = it % kOzStages;
                        if (!mbar_wait(&full[s], (it / kOzStages) & 1u)) atomicCAS(P.err, 0, KORE_DEVERR_FLAG);
                        oz_fence_after();
                        const uint64_t da = core_desc(smem_u32(smem + (size_t)s * kOzStage));
                        const uint64_t db = core_desc(smem_u32(smem + (size_t)s * kOzStage + kOzStepA));
                        // descriptor steps: slice 2 x part, part Im after Re
                        constexpr uint64_t sa = kOzSliceA >> 4, sb = kOzSliceB >> 4;
                        for (int q = 0; q < 3; ++q) {
                            const int d = 8 - 3 * g - q;
                            const uint32_t re = tmem + (uint32_t)(q * 2 * kOzN), im = re + kOzN;
                            for (int i = 0; i <= d; ++i) {
                                const uint64_t ar = da + i * sa, ai = ar + sa / 2;
                                const uint64_t br = db + (d - i) * sb, bi = br + sb / 2;
                                const uint32_t acc = (k == k0 && i == 0) ? 0u : 1u;
                                oz_mma(re, ar, br, f16_idesc(0), acc);
                                oz_mma(im, ar, bi, f16_idesc(0), acc);
                                oz_mma(re, ai, bi, f16_idesc(1), 1u);
                                oz_mma(im, ai, br, f16_idesc(0), 1u);
                            }
                        }
                        oz_commit(&empty[s]);
                    }
                    oz_commit(accum);
                }
            }
        }
        __syncwarp();
    } else {
        // rows 32 (warp % 4) .. + 31 (the tensor-memory lanes this warp reaches), columns
        // 16 (warp / 4) .. + 15 of the tile
        const int row = mt * kOzM + (warp & 3) * 32 + lane, cb = (warp >> 2) * 16;
        const uint32_t tl = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)cb;
        uint32_t pass = 0;
        for (int sg = 0; sg < nseg; ++sg) {
            const int prod = sg / parts, part = sg - prod * parts;
            const int n = (part + 1) * steps / parts - part * steps / parts;
            long long gr[16], gi[16];   // sums of d = 3 .. 8 in units of 128^-10, below 2^61
#pragma unroll
            for (int c = 0; c < 16; ++c) gr[c] = gi[c] = 0;
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                const int np = CUT ? oz_pieces(n, g) : 1;
                for (int p = 0; p < np; ++p, ++pass) {
                    if (!mbar_wait(accum, pass & 1u)) atomicCAS(P.err, 0, KORE_DEVERR_FLAG);
                    oz_fence_after();
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
                        const int sh = kOzBits * (3 * g + q);
#pragma unroll
                        for (int h = 0; h < 16; h += 8) {
                            float vr[8], vi[8];
                            oz_ld8(tl + (uint32_t)(q * 2 * kOzN + h), vr);
                            oz_ld8(tl + (uint32_t)(q * 2 * kOzN + kOzN + h), vi);
                            oz_ld_wait();
#pragma unroll
                            for (int c = 0; c < 8; ++c) {
                                gr[h + c] += (long long)__float2int_rn(vr[c]) << sh;
                                gi[h + c] += (long long)__float2int_rn(vi[c]) << sh;
                            }
                        }
                    }
                    oz_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(drained);
                }
            }
            if (!mbar_wait(accum, pass & 1u)) atomicCAS(P.err, 0, KORE_DEVERR_FLAG);
            oz_fence_after();
            const int *ea = P.ea + (int64_t)(prod ? job.a2 : job.a1) * S, *eb = P.eb + (int64_t)(prod ? job.b2 : job.b1) * ncols;
            const int er = row < S ? ea[row] : kOzNone;
            const bool add = sg > 0 || job.beta;
            // the group update reads its source, zero in the group's pivot rows
            const double2 *old_c = job.C;
            bool keep = row < S;
            if (GROUP) {
                old_c = P.group.source(blockIdx.y);
                const int u = row < S ? P.group.used[P.group.rows(blockIdx.y) + row] : 0;
                keep = keep && !(u > P.group.g0 && u <= P.group.g1);
            }
#pragma unroll
            for (int h = 0; h < 16; h += 4) {
                // d = 2, 1, 0 in units of 128^-4; four columns at a time
                long long tr[4], ti[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) tr[c] = ti[c] = 0;
                uint32_t r[3][2][4];
#pragma unroll
                for (int q = 0; q < 3; ++q)
#pragma unroll
                    for (int z = 0; z < 2; ++z)
                        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                                     : "=r"(r[q][z][0]), "=r"(r[q][z][1]), "=r"(r[q][z][2]), "=r"(r[q][z][3])
                                     : "r"(tl + (uint32_t)(q * 2 * kOzN + z * kOzN + h))
                                     : "memory");
                oz_ld_wait();
#pragma unroll
                for (int q = 0; q < 3; ++q)
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        tr[c] += (long long)__float2int_rn(__uint_as_float(r[q][0][c])) << (kOzBits * q);
                        ti[c] += (long long)__float2int_rn(__uint_as_float(r[q][1][c])) << (kOzBits * q);
                    }
                double2 old[4];
                const int col0 = nt * kOzN + cb + h;
                int64_t at[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    at[c] = row + (int64_t)(GROUP ? P.group.column(col0 + c) : col0 + c) * S;
                    old[c] = (add && keep && col0 + c < ncols) ? old_c[at[c]] : mk(0.0, 0.0);
                }
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (row < S && col0 + c < ncols) {
                        const int ec = eb[col0 + c];
                        double2 v;
                        if (er == kOzBad || ec == kOzBad) v = mk(NAN, NAN);
                        else if (er == kOzNone || ec == kOzNone) v = mk(0.0, 0.0);
                        else v = mk(from_digits(tr[c], gr[h + c], er + ec), from_digits(ti[c], gi[h + c], er + ec));
                        if (job.negate) v = -v;
                        job.C[at[c]] = add ? old[c] + v : v;
                    }
            }
            oz_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(drained);
            ++pass;
        }
    }
    oz_fence_before();
    __syncthreads();
    if (warp == kOzEpiWarps + 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// Operands and jobs of one batch, and its place in the workspace.
struct OzBatch {
    std::vector<OzPair> pairs;
    std::vector<OzOperand> a, b;
    std::vector<OzJob> jobs;
    void clear() { pairs.clear(); a.clear(); b.clear(); jobs.clear(); }
};

int64_t round256(int64_t x) { return (x + 255) & ~(int64_t)255; }

// workspace bytes of a batch of np pairs, na and nb operands and nj jobs
int64_t oz_batch_bytes(int S, int64_t np, int64_t na, int64_t nb, int64_t nj) {
    return round256(na * oz_bytes_a(S, S)) + round256(nb * oz_bytes_b(S, S)) + round256((np + na + nb) * S * 4) +
           round256(np * sizeof(OzPair)) + round256((na + nb) * sizeof(OzOperand)) + round256(nj * sizeof(OzJob));
}

int oz_run(cudaStream_t st, int device, int S, const OzBatch &w, unsigned char *ws, int *err) {
    if (w.jobs.empty()) return KORE_OK;
    const int64_t np = (int64_t)w.pairs.size(), na = (int64_t)w.a.size(), nb = (int64_t)w.b.size();
    unsigned char *pa = ws, *pb = pa + round256(na * oz_bytes_a(S, S));
    int *rho = reinterpret_cast<int *>(pb + round256(nb * oz_bytes_b(S, S)));
    int *ea = rho + np * S, *eb = ea + na * S;
    unsigned char *tab = reinterpret_cast<unsigned char *>(rho) + round256((np + na + nb) * S * 4);
    // one upload of the tables
    std::vector<unsigned char> h(round256(np * sizeof(OzPair)) + round256((na + nb) * sizeof(OzOperand)) +
                                 w.jobs.size() * sizeof(OzJob));
    auto put = [&](size_t at, const void *src, size_t n) { if (n) memcpy(h.data() + at, src, n); };
    const size_t at_ops = round256(np * sizeof(OzPair)), at_jobs = at_ops + round256((na + nb) * sizeof(OzOperand));
    put(0, w.pairs.data(), np * sizeof(OzPair));
    put(at_ops, w.a.data(), na * sizeof(OzOperand));
    put(at_ops + na * sizeof(OzOperand), w.b.data(), nb * sizeof(OzOperand));
    put(at_jobs, w.jobs.data(), w.jobs.size() * sizeof(OzJob));
    KORE_CUDA_TRY(cudaMemcpyAsync(tab, h.data(), h.size(), cudaMemcpyHostToDevice, st));
    const OzOperand *da = reinterpret_cast<const OzOperand *>(tab + at_ops);
    k_oz_rho<<<dim3(kore_div_up(S, 32), (unsigned)np), 256, 0, st>>>(reinterpret_cast<const OzPair *>(tab), S, rho);
    k_oz_split_a<<<dim3(kore_div_up(S, 32), (unsigned)na), 256, 0, st>>>(da, S, rho, pa, oz_bytes_a(S, S), ea);
    k_oz_split_b<<<dim3(kore_div_up(S, 8), (unsigned)nb), 256, 0, st>>>(da + na, S, rho, pb, oz_bytes_b(S, S), eb);
    OzParams P{};
    P.jobs = reinterpret_cast<const OzJob *>(tab + at_jobs);
    P.pa = pa; P.pb = pb; P.ea = ea; P.eb = eb;
    P.bytes_a = oz_bytes_a(S, S); P.bytes_b = oz_bytes_b(S, S);
    P.S = S; P.nt = oz_nt(S); P.steps = oz_steps(S); P.err = err;
    auto gemm = P.steps > kOzPlainSteps ? k_oz_gemm<false, true> : k_oz_gemm<false, false>;
    KORE_TRY(kore_allow_max_dyn_smem(gemm, device));
    gemm<<<dim3(oz_mt(S) * oz_nt(S), (unsigned)w.jobs.size()), kOzThreads, kOzSmem, st>>>(P);
    KORE_LAUNCHED(4);
    KORE_CUDA_TRY(cudaGetLastError());
    return KORE_OK;
}

}  // namespace

// ----------------------------------------------------------------------------- factorisation use
// The products run in batches that share a workspace of at most 512 MB (several waves of
// tiles at the largest blocks; the planes take 2.3 times the matrices).
constexpr int64_t kOzWorkspace = 512ll << 20;

// workspace bytes of one block's group update, W columns
static int64_t oz_group_bytes(int S, int W) {
    return oz_bytes_a(S, W) + oz_bytes_b(S, W) + round256((int64_t)(W + 2 * S) * 4);
}

int64_t kore_oz_workspace_bytes(int S, int64_t K, int64_t cap) {
    int64_t need = 0;
    for (int64_t Kl = K - K / 2; Kl > 1; Kl -= Kl / 2) {   // levels >= 1
        const int64_t no = Kl / 2 * cap, ne = (Kl - Kl / 2) * cap;
        need = std::max({need, oz_batch_bytes(S, no, no, 2 * no, 2 * no),
                         oz_batch_bytes(S, no, 2 * ne, 2 * no, 3 * ne)});
    }
    // the group updates of the eliminated blocks of level 0 (a group has at most 64 columns)
    const int64_t group = std::max<int64_t>(K / 2, 1) * cap * oz_group_bytes(S, 64);
    // one block's products always fit
    return std::max(std::min(std::max(need, group), kOzWorkspace), oz_batch_bytes(S, 2, 2, 4, 3));
}

namespace {

struct OzQueue {
    kore_plan *p;
    OzBatch w;
    // room for a unit of np pairs, na and nb operands and nj jobs: runs the batch when it
    // would not fit with it
    int room(int64_t np, int64_t na, int64_t nb, int64_t nj, bool *flushed) {
        *flushed = false;
        if (oz_batch_bytes(p->S, (int64_t)w.pairs.size() + np, (int64_t)w.a.size() + na, (int64_t)w.b.size() + nb,
                           (int64_t)w.jobs.size() + nj) <= p->oz_bytes)
            return KORE_OK;
        *flushed = true;
        return run();
    }
    int run() {
        KORE_TRY(oz_run(p->stream, p->device, p->S, w, static_cast<unsigned char *>(p->d_oz), p->d_err));
        w.clear();
        return KORE_OK;
    }
    int pair(const double2 *x0, const double2 *x1) {
        w.pairs.push_back({x0, x1});
        return (int)w.pairs.size() - 1;
    }
    int a(const double2 *x, int pr) {
        w.a.push_back({x, pr});
        return (int)w.a.size() - 1;
    }
    int b(const double2 *x, int pr) {
        w.b.push_back({x, pr});
        return (int)w.b.size() - 1;
    }
};

}  // namespace

// G_j = D_j^-1 L_q and H_j = D_j^-1 U_q of the odd blocks of a level >= 1 (complex128).
int kore_gh_update_oz(kore_plan *p, const BcrLevel &lv) {
    const int64_t SS = (int64_t)p->S * p->S;
    OzQueue z{p, {}};
    bool flushed;
    for (int sh = p->fw_lo; sh < p->fw_lo + p->fw_n; ++sh) {
        const double2 *LU = static_cast<const double2 *>(p->d_LU) + sh * p->lu_stride();
        const int64_t f = sh * p->f_stride();
        for (int o = 0; o < lv.nodd; ++o) {
            const int64_t q = 2 * o + 1, j = f + q * lv.stride * SS;
            const bool hasr = q + 1 < lv.Kl;   // no right neighbour: H_j is never read
            const double2 *L = LU + (lv.lu_L + q) * SS, *U = hasr ? LU + (lv.lu_U + q) * SS : nullptr;
            KORE_TRY(z.room(1, 1, 2, 2, &flushed));
            const int pr = z.pair(L, U), a = z.a(static_cast<const double2 *>(p->d_Dinv) + j, pr);
            z.w.jobs.push_back({a, z.b(L, pr), -1, -1, static_cast<double2 *>(p->d_Gm) + j, 0, 0});
            if (hasr) z.w.jobs.push_back({a, z.b(U, pr), -1, -1, static_cast<double2 *>(p->d_Hm) + j, 0, 0});
        }
    }
    return z.run();
}

// Even-block update of a level >= 1 (complex128): D_i -= L_q H_jl + U_q G_jr; L' = -L_q G_jl;
// U' = -U_q H_jr.
int kore_even_update_oz(kore_plan *p, const BcrLevel &lv) {
    const int64_t SS = (int64_t)p->S * p->S;
    OzQueue z{p, {}};
    bool flushed;
    for (int sh = p->fw_lo; sh < p->fw_lo + p->fw_n; ++sh) {
        double2 *LU = static_cast<double2 *>(p->d_LU) + sh * p->lu_stride();
        double2 *Dw = static_cast<double2 *>(p->d_Dw) + sh * p->f_stride();
        const double2 *G = static_cast<const double2 *>(p->d_Gm) + sh * p->f_stride();
        const double2 *H = static_cast<const double2 *>(p->d_Hm) + sh * p->f_stride();
        // the split G and H of the last odd block queued: the left neighbour of the next even one
        int opr = -1, og = -1, oh = -1;
        auto odd = [&](int64_t q) {   // position q
            const int64_t j = q * lv.stride * SS;
            const bool hasr = q + 1 < lv.Kl;
            opr = z.pair(G + j, hasr ? H + j : nullptr);
            og = z.b(G + j, opr);
            oh = hasr ? z.b(H + j, opr) : -1;
        };
        for (int e = 0; e < lv.neven; ++e) {
            const int64_t q = 2 * e;
            const bool hasl = q >= 1, hasr = q + 1 < lv.Kl;
            KORE_TRY(z.room(2, 2, 4, 3, &flushed));
            OzJob d{-1, -1, -1, -1, Dw + q * lv.stride * SS, 1, 1};
            if (hasl) {
                if (flushed || opr < 0) odd(q - 1);
                const int a = z.a(LU + (lv.lu_L + q) * SS, opr);
                d.a1 = a;
                d.b1 = oh;
                if (lv.lu_nL >= 0) z.w.jobs.push_back({a, og, -1, -1, LU + (lv.lu_nL + e) * SS, 1, 0});
            }
            if (hasr) {
                odd(q + 1);
                const int a = z.a(LU + (lv.lu_U + q) * SS, opr);
                (hasl ? d.a2 : d.a1) = a;
                (hasl ? d.b2 : d.b1) = og;
                if (lv.lu_nU >= 0 && q + 2 < lv.Kl) z.w.jobs.push_back({a, oh, -1, -1, LU + (lv.lu_nU + e) * SS, 1, 0});
            }
            if (hasl || hasr) z.w.jobs.push_back(d);
        }
    }
    return z.run();
}

int kore_group_update_oz(kore_plan *p, const BcrLevel &lv, int nodd, int g0, int g1) {
    const int S = p->S, W = g1 - g0, n = S - W;
    const int64_t lo = p->fw_lo;
    OzGroup q{static_cast<double2 *>(p->d_T) + lo * p->t_stride(), static_cast<const double2 *>(p->d_Dw) + lo * p->f_stride(),
              p->d_piv + lo * p->p_stride(), p->d_used + lo * p->p_stride(), p->t_stride(), p->t_block(sizeof(double2)),
              p->f_stride(), p->p_stride(), nodd, lv.stride, S, g0, g1, 0};
    const int total = nodd * p->fw_n;
    const int per = (int)std::min<int64_t>(std::min(total, 65535), p->oz_bytes / oz_group_bytes(S, W));
    if (per < 1 || oz_steps(W) > kOzPlainSteps) return KORE_EINVAL;
    KORE_TRY(kore_allow_max_dyn_smem(k_oz_gemm<true, false>, p->device));
    for (q.first = 0; q.first < total; q.first += per) {
        const int nb = std::min(per, total - q.first);
        unsigned char *pa = static_cast<unsigned char *>(p->d_oz), *pb = pa + nb * oz_bytes_a(S, W);
        int *rho = reinterpret_cast<int *>(pb + nb * oz_bytes_b(S, W)), *ea = rho + (int64_t)nb * W,
            *eb = ea + (int64_t)nb * S;
        k_oz_group_rho<<<nb, 512, 0, p->stream>>>(q, rho);
        k_oz_group_a<<<dim3(kore_div_up(S, 32), nb), 256, 0, p->stream>>>(q, rho, pa, oz_bytes_a(S, W), ea);
        k_oz_group_b<<<dim3(kore_div_up(n, 8), nb), 256, 0, p->stream>>>(q, rho, pb, oz_bytes_b(S, W), eb);
        OzParams P{};
        P.pa = pa; P.pb = pb; P.ea = ea; P.eb = eb;
        P.bytes_a = oz_bytes_a(S, W); P.bytes_b = oz_bytes_b(S, W);
        P.S = S; P.nt = oz_nt(n); P.steps = oz_steps(W); P.err = p->d_err; P.group = q;
        k_oz_gemm<true, false><<<dim3(oz_mt(S) * P.nt, nb), kOzThreads, kOzSmem, p->stream>>>(P);
        KORE_LAUNCHED(4);
    }
    KORE_CUDA_TRY(cudaGetLastError());
    return KORE_OK;
}

extern "C" int kore_oz_selftest(int device, int S, const double *A1, const double *B1, const double *A2, const double *B2,
                                double *C, int negate, int beta) {
    if (S <= 0 || S > 1024 || !A1 || !B1 || !C || !A2 != !B2) return KORE_EINVAL;
    int prev = -1;
    cudaGetDevice(&prev);
    KORE_CUDA_TRY(cudaSetDevice(device));
    const size_t SS = (size_t)S * S, bytes = SS * sizeof(double2);
    const double *host[] = {A1, B1, A2, B2, C};
    double2 *m = nullptr;   // A1, B1, A2, B2, C
    unsigned char *ws = nullptr;
    int *flag = nullptr;
    int rc = KORE_OK;
    auto ck = [&](cudaError_t e) { if (e != cudaSuccess && rc == KORE_OK) rc = (e == cudaErrorMemoryAllocation) ? KORE_ENOMEM : KORE_ECUDA; };
    ck(cudaMalloc(&m, 5 * bytes));
    ck(cudaMalloc(&ws, oz_batch_bytes(S, 2, 2, 2, 1)));
    ck(cudaMalloc(&flag, sizeof(int)));
    if (rc == KORE_OK) {
        for (int i = 0; i < 5; ++i)
            if (host[i]) ck(cudaMemcpy(m + i * SS, host[i], bytes, cudaMemcpyHostToDevice));
        ck(cudaMemset(flag, 0, sizeof(int)));
        OzBatch w;
        for (int q = 0; q < (A2 ? 2 : 1); ++q) {
            w.pairs.push_back({m + (2 * q + 1) * SS, nullptr});
            w.a.push_back({m + 2 * q * SS, q});
            w.b.push_back({m + (2 * q + 1) * SS, q});
        }
        w.jobs.push_back({0, 0, A2 ? 1 : -1, A2 ? 1 : -1, m + 4 * SS, negate != 0, beta != 0});
        if (rc == KORE_OK) rc = oz_run(0, device, S, w, ws, flag);
        int h = 0;
        if (rc == KORE_OK) {
            ck(cudaMemcpy(&h, flag, sizeof(int), cudaMemcpyDeviceToHost));
            ck(cudaMemcpy(C, m + 4 * SS, bytes, cudaMemcpyDeviceToHost));
            if (rc == KORE_OK && h != 0) rc = KORE_ETIMEOUT;
        }
    }
    cudaFree(m); cudaFree(ws); cudaFree(flag);
    if (prev >= 0) cudaSetDevice(prev);
    return rc;
}
