// Factorisation of A - sigma*B by block cyclic reduction over the l-major blocks.
//
// The row-equilibrated pencil R(A - sigma B) is block tridiagonal with diagonal
// blocks D_i and couplings L_i (to block i-1) and U_i (to block i+1).  One reduction
// level eliminates the blocks at odd positions j of the active sequence:
//
//          D_j^-1 by Gauss-Jordan,   G_j = D_j^-1 L_j,   H_j = D_j^-1 U_j
//     for the even neighbours i (odd neighbours jl = left, jr = right):
//          D_i <- D_i - L_i H_jl - U_i G_jr
//          L_i <- -L_i G_jl        (couples i to the even block left of jl)
//          U_i <- -U_i H_jr        (couples i to the even block right of jr)
//
// which halves the number of active blocks; after ceil(log2 K) levels one block is
// left and only its inverse is formed.  All blocks of a level are independent, so
// every kernel below is batched over the blocks of the level: the work of one
// factorisation is a few hundred launches of GPU-wide batched dense kernels instead
// of a chain of K dependent block steps.  Level 0 takes D, L, U from the CSR
// (L and U sparse: the even-block update is a sparse x dense product); the dense
// updates of the higher levels are batched complex GEMMs.
//
// Gauss-Jordan is blocked and in place: one CTA per block reduces a panel of NB columns
// in registers (pivot search over the rows not yet used as pivots, elimination that turns
// the panel into the columns of the accumulated elementary transform E), then every other
// column t of the block is updated by t <- E t, i.e. t[r] += sum_c E[r,c] t[piv_c], with
// the pivot rows themselves replaced.  The columns left of the panel are then columns of
// the inverse built so far (E applied to the columns of the identity that an [D | I] work
// matrix would carry), so the work matrix is S x S and a block costs 8 S^3 real operations
// instead of 12.  Rows are never swapped: the pivot row of column k is recorded and the
// inverse is gathered by it.  Pivoting stays inside each diagonal block.
//
// Many shifts (forcing frequencies, targets) of one pencil are factorised together:
// every kernel carries the shift as one more grid dimension, and shift s uses its own
// row scales and factor set at offset s * stride.
//
// This replaces the sparse LU that SLEPc's ST sinvert / PETSc's PCLU build inside
// bin/solve.py:123 and :227; the ordering (odd-even elimination of l-blocks) is what
// exposes the parallelism.
#include "kore_internal.cuh"
#include <climits>
#include <algorithm>

namespace {

// Device view of the plan for the factorisation kernels; shift s uses offset
// s * (f|lu|t|p|rs)_stride into the per-shift buffers.
template <typename C>
struct FV {
    int S, K;
    int64_t np;
    const int *arow, *acol, *asplit, *brow, *bcol, *bsz;
    const double2 *aval;
    const double *bval;
    int has_b;
    const double2 *sigma;
    double *rscale;
    C *Dinv, *G, *H, *Dw, *LU, *T;
    int *piv, *used, *err;
    const int *cc_ptr, *cc_row, *cc_src;
    const int *ell_col;      // level-0 coupling rows of every block (kore_plan::d_ell_*)
    const C *ell_val;
    int ell_w;
    int64_t ell_stride;
    int64_t f_stride, lu_stride, t_stride, t_block, p_stride;
};

// View of the plan's factor storage starting at the factor window's first shift (shift
// fw_lo + s of the plan is shift s of the view).
template <typename C>
FV<C> make_fv(kore_plan *p) {
    FV<C> v;
    const int64_t lo = p->fw_lo;
    v.S = p->S; v.K = p->K; v.np = p->np;
    v.arow = p->d_arow; v.acol = p->d_acol; v.asplit = p->d_asplit; v.brow = p->d_brow; v.bcol = p->d_bcol;
    v.bsz = p->d_bsz; v.aval = p->d_aval; v.bval = p->d_bval; v.has_b = p->has_b ? 1 : 0;
    v.sigma = p->d_sigma + lo; v.rscale = p->d_rscale + lo * p->np;
    v.Dinv = static_cast<C *>(p->d_Dinv) + lo * p->f_stride(); v.G = static_cast<C *>(p->d_Gm) + lo * p->f_stride();
    v.H = static_cast<C *>(p->d_Hm) + lo * p->f_stride(); v.Dw = static_cast<C *>(p->d_Dw) + lo * p->f_stride();
    v.LU = static_cast<C *>(p->d_LU) + lo * p->lu_stride(); v.T = static_cast<C *>(p->d_T) + lo * p->t_stride();
    v.piv = p->d_piv + lo * p->p_stride();
    v.used = p->d_used + lo * p->p_stride(); v.err = p->d_err;
    v.cc_ptr = p->d_cc_ptr; v.cc_row = p->d_cc_row; v.cc_src = p->d_cc_src;
    v.ell_col = p->d_ell_col; v.ell_val = static_cast<const C *>(p->d_ell_val) + lo * p->ell_stride();
    v.ell_w = p->ell_w;
    v.ell_stride = p->ell_stride();
    v.f_stride = p->f_stride(); v.lu_stride = p->lu_stride(); v.t_stride = p->t_stride(); v.t_block = p->t_block(sizeof(C)); v.p_stride = p->p_stride();
    return v;
}

// Row equilibration by powers of two (exact): rscale[p] = 2^-e with
// e = exponent of max(max_e |a_pe|, |sigma| max_e |b_pe|); also the row 1-norms of
// |A| + |sigma||B| whose maximum bounds ||A - sigma B||_inf.  The entries are read once for
// all shifts (one thread per row; their square roots run on the FP64 pipe).  Per-CTA maxima
// to red[s * gridDim.x + blockIdx.x].
template <typename C>
__global__ void __launch_bounds__(256) k_rowinfo(FV<C> v, int nshift, double *__restrict__ red) {
    __shared__ double sm[8];
    const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    double amax = 0.0, asum = 0.0, bmax = 0.0, bsum = 0.0;
    if (p < v.np) {
        const int a1 = v.arow[p + 1];
#pragma unroll 4
        for (int e = v.arow[p]; e < a1; ++e) {
            const double2 a = v.aval[e];
            const double t = a.y == 0.0 ? fabs(a.x) : a.x == 0.0 ? fabs(a.y) : sqrt(abs2(a));
            amax = fmax(amax, t);
            asum += t;
        }
        if (v.has_b) {
            const int b1 = v.brow[p + 1];
#pragma unroll 4
            for (int e = v.brow[p]; e < b1; ++e) {
                const double t = fabs(v.bval[e]);
                bmax = fmax(bmax, t);
                bsum += t;
            }
        }
    }
    for (int s = 0; s < nshift; ++s) {
        const double sabs = sqrt(abs2(v.sigma[s]));
        double mx = 0.0;
        if (p < v.np) {
            const double am = fmax(amax, sabs * bmax);
            v.rscale[(int64_t)s * v.np + p] = (am > 0.0) ? ldexp(1.0, -ilogb(am)) : 1.0;
            mx = asum + sabs * bsum;
        }
        mx = warp_max_d(mx);
        if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = mx;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < 8; ++w) mx = fmax(mx, sm[w]);
            red[(int64_t)s * gridDim.x + blockIdx.x] = mx;
        }
        __syncthreads();
    }
}

// minf[s] = max of red[s * n .. s * n + n), one CTA per shift
__global__ void k_minf(const double *__restrict__ red, int n, double *__restrict__ minf) {
    __shared__ double sm[8];
    double mx = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) mx = fmax(mx, red[(int64_t)blockIdx.x * n + i]);
    mx = warp_max_d(mx);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) mx = fmax(mx, sm[w]);
        minf[blockIdx.x] = mx;
    }
}

// Values of the padded level-0 coupling rows for every shift: rscale_row * A entry in
// the factor precision (grid (x, shift)).
template <typename C>
__global__ void k_ell_fill(int64_t ell_stride, int ell_w, int ntile, int S, int64_t np,
                           const int *__restrict__ src, const double2 *__restrict__ aval,
                           const double *__restrict__ rscale, C *__restrict__ val) {
    const int64_t s = blockIdx.y;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < ell_stride;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int e = src[idx];
        C v = czero<C>();
        if (e >= 0) {
            const int64_t lane = idx & 31, tile = idx / 32 / ell_w;   // tile = block * ntile + t
            const int64_t bi = tile / ntile, t = tile - bi * ntile;
            const int64_t row = bi * S + t * 32 + lane;
            v = from_c128<C>(rscale[s * np + row] * aval[e]);
        }
        val[s * ell_stride + idx] = v;
    }
}

// Dw <- 0 with the identity on the padded diagonal of every block, all shifts.
template <typename C>
__global__ void k_Dw_init(FV<C> v, int nshift) {
    const int64_t SS = (int64_t)v.S * v.S, per = (int64_t)v.K * SS, total = per * nshift;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t w = idx % per;
        const int64_t i = w / SS;
        const int64_t e = w - i * SS;
        const int c = (int)(e / v.S), r = (int)(e - (int64_t)c * v.S);
        v.Dw[idx] = (r == c && r >= v.bsz[i]) ? cone<C>() : czero<C>();
    }
}

// One warp per (shift, row): Dw_i[r, :] = rs_r (D_i - sigma B_i)[r, :] from the CSR.
// A and B entries of the same column are combined in FP64 and rounded once.
template <typename C>
__global__ void k_Dw_scatter(FV<C> v, int nshift) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int S = v.S;
    for (int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; w < v.np * nshift; w += nw) {
        const int64_t s = w / v.np, p = w - s * v.np;
        const int64_t i = p / S;
        const int r = (int)(p - i * S);
        const double2 sigma = v.sigma[s];
        const double rs = v.rscale[s * v.np + p];
        C *D = v.Dw + s * v.f_stride + i * (int64_t)S * S;
        const int eD = v.asplit[2 * p], eU = v.asplit[2 * p + 1];
        for (int e = eD + lane; e < eU; e += 32) D[r + (int64_t)(v.acol[e] - i * S) * S] = from_c128<C>(rs * v.aval[e]);
        __syncwarp();
        if (v.has_b)
            for (int e = v.brow[p] + lane; e < v.brow[p + 1]; e += 32) {
                const int c = v.bcol[e];
                int lo = eD, hi = eU;   // matching A entry: binary search in the sorted D segment
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (v.acol[mid] < c) lo = mid + 1; else hi = mid;
                }
                const double2 a = (lo < eU && v.acol[lo] == c) ? v.aval[lo] : mk(0.0, 0.0);
                D[r + (int64_t)(c - i * S) * S] = from_c128<C>(rs * (a - v.bval[e] * sigma));
            }
    }
}

// Pivot keys: |x|^2 as the bits of a non-negative number, whose integer order is the
// numeric one, so the search runs on the integer units (on this GPU an FP64 comparison
// costs as much as an FP64 product).  0 (a zero, a NaN or a used row) is never a pivot.
__device__ __forceinline__ unsigned long long pivot_key(float2 x) {
    const float v = abs2(x);
    return v > 0.f ? (unsigned long long)__float_as_uint(v) : 0ull;
}
__device__ __forceinline__ unsigned long long pivot_key(double2 x) {
    const double v = abs2(x);
    const long long b = __double_as_longlong(v);
    return (b > 0 && b <= 0x7ff0000000000000ll) ? (unsigned long long)b : 0ull;   // +0, NaN: 0
}
// 1 / x.  complex128: conj(x) / |x|^2 of x scaled by a power of two to magnitude [1, 4), one
// FP64 division (about a dozen steps of the pipe each) where the scaled quotient takes three.
__device__ __forceinline__ float2 inverse(float2 x) { return cdiv(cone<float2>(), x); }
__device__ __forceinline__ double2 inverse(double2 x) {
    const int hx = (__double2hiint(x.x) >> 20) & 0x7ff, hy = (__double2hiint(x.y) >> 20) & 0x7ff;
    const int e = max(hx, hy);
    if (e < 64 || e > 1982) return cdiv(cone<double2>(), x);   // 2^-e itself near the range's ends
    const double s = __hiloint2double((2046 - e) << 20, 0);    // 2^(1023 - e)
    const double2 z = s * x;
    const double r = 1.0 / abs2(z);
    return mk(s * (z.x * r), -(s * (z.y * r)));
}
// The largest key of a warp and the lowest lane that holds it.
template <typename C>
__device__ __forceinline__ unsigned long long warp_argmax(unsigned long long key, int &lane_of) {
    const unsigned lo = (unsigned)key;
    if (sizeof(C) == 8) {
        const unsigned m = __reduce_max_sync(0xffffffffu, lo);
        lane_of = __ffs(__ballot_sync(0xffffffffu, lo == m)) - 1;
        return m;
    }
    const unsigned hi = (unsigned)(key >> 32);
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned l2 = hi == mh ? lo : 0u;
    const unsigned ml = __reduce_max_sync(0xffffffffu, l2);
    lane_of = __ffs(__ballot_sync(0xffffffffu, hi == mh && lo == ml)) - 1;
    return ((unsigned long long)mh << 32) | ml;
}

// The diagonal block that work matrix o of shift sh inverts: the odd block at position
// 2 o + 1 of a level (original block (2 o + 1) stride), or with stride 0 block 0, the top
// of the reduction.
template <typename C>
__device__ __forceinline__ const C *diag_block(const FV<C> &v, int64_t o, int64_t sh, int stride) {
    return v.Dw + sh * v.f_stride + (2 * o + 1) * stride * (int64_t)v.S * v.S;
}

// Panel reduction of columns [k0, k0+nb) of T_o; one CTA per (odd block o = blockIdx.x,
// shift = blockIdx.y), one thread per row, which holds its NB entries of the panel in
// registers.  Every elimination step works on register 0 and shifts the others down by
// one, the finished column of E entering at the top: after nb steps column j of the
// panel is register NB - nb + j, and the loop body needs no indexed registers.
// The panel is a chain of S dependent steps per block: with the panel in shared memory,
// one step cost four barriers, an FP64 pivot search and two shared-memory accesses per
// product; here it is two barriers, an integer search and one broadcast load per two
// columns.  The first panel and its update
// read the diagonal block itself, which stays as it is.
// With Helper (up to 512 rows) one more warp shortens the chain: a step updates the next
// pivot column first and hands its candidates over, and while the row warps update the
// other columns the helper picks the pivot and inverts it (60 blocks of 96 in complex128,
// factorised and solved: 5.20 -> 4.86 ms; two shifts of the MAC shell, S = 360, in complex64:
// 9.58 -> 9.37 ms).
__device__ __forceinline__ void bar_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int threads) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
constexpr int panel_threads(int rows) { return rows <= 512 ? rows + 32 : rows; }

template <typename C, int NB, int MAXT>
__global__ void __launch_bounds__(panel_threads(MAXT)) k_panel(FV<C> v, int k0, int nb, int stride) {
    constexpr bool Helper = MAXT <= 512;
    __shared__ __align__(16) C prow[NB];
    __shared__ __align__(16) C wval[32];
    __shared__ C s_inv;
    __shared__ unsigned long long wkey[32];
    __shared__ int wrow[32];
    __shared__ int s_piv[NB], s_p;
    const int S = v.S;
    const int64_t o = blockIdx.x, sh = blockIdx.y;
    C *T = v.T + sh * v.t_stride + o * v.t_block + (int64_t)k0 * S;
    const C *src = k0 == 0 ? diag_block(v, o, sh, stride) : T;
    int *piv = v.piv + sh * v.p_stride + o * S;
    int *used = v.used + sh * v.p_stride + o * S;
    const int threads = blockDim.x;
    const int r = threadIdx.x, lane = r & 31, w = r >> 5, nw = (threads >> 5) - (Helper ? 1 : 0);
    after_previous();

    // the largest candidate: its row, or -1 when there is none; with inv also its inverse
    auto choose = [&](C *inv) {
        int wl;
        const unsigned long long best = warp_argmax<C>(lane < nw ? wkey[lane] : 0ull, wl);
        if (best == 0ull) return -1;
        if (inv) *inv = inverse(wval[wl]);
        return wrow[wl];
    };
    if (Helper && w == nw) {
        for (int c = 0; c < nb; ++c) {
            bar_sync(1, threads);   // the candidates of column c
            C inv = czero<C>();
            const int p = choose(&inv);
            if (lane == 0) {
                s_p = p;
                s_inv = inv;
            }
            bar_sync(0, threads);
            if (p < 0) break;
            bar_sync(0, threads);
        }
        return;
    }

    const bool in = r < S;
    C P[NB];
#pragma unroll
    for (int c = 0; c < NB; ++c) P[c] = (in && c < nb) ? src[r + (int64_t)c * S] : czero<C>();
    int mine = (in && k0 != 0) ? used[r] : 0;   // 1 + the column this row is the pivot of, or 0
    bool u = !in || mine != 0;
    auto propose = [&](C x) {   // this warp's candidate for the next pivot
        int l;
        const unsigned long long k = warp_argmax<C>(u ? 0ull : pivot_key(x), l);
        if (lane == l) {
            wkey[w] = k;
            wrow[w] = r;
            wval[w] = x;
        }
        if (Helper) bar_arrive(1, threads);
    };
    propose(P[0]);
    int c = 0;
    for (; c < nb; ++c) {
        bar_sync(0, threads);
        const int p = Helper ? s_p : choose(nullptr);
        if (p < 0) {   // uniform over the CTA
            if (r == 0) atomicCAS(v.err, 0, KORE_DEVERR_PIVOT);
            break;
        }
        if (w == p >> 5) {   // the pivot row's warp publishes the row, scaled by 1 / pivot
            if (r == p) {
                u = true;
                mine = k0 + c + 1;
                s_piv[c] = p;
#pragma unroll
                for (int q = 0; q < NB; ++q) prow[q] = P[q];
            }
            __syncwarp();
            const C dinv = Helper ? s_inv : inverse(prow[0]);
            const C own = lane < NB ? prow[lane] : czero<C>();
            __syncwarp();
            if (lane < NB) prow[lane] = lane == 0 ? dinv : own * dinv;
        }
        bar_sync(0, threads);
        const C dinv = prow[0], mult = P[0];
        P[0] = r == p ? prow[1] : cfms(P[1], mult, prow[1]);
        if (c + 1 < nb) propose(P[0]);
        if (r == p) {
#pragma unroll
            for (int q = 2; q < NB; ++q) P[q - 1] = prow[q];
            P[NB - 1] = dinv;
        } else {
#pragma unroll
            for (int q = 2; q < NB; ++q) P[q - 1] = cfms(P[q], mult, prow[q]);
            P[NB - 1] = -(mult * dinv);
        }
    }
    before_next();
    const int done = c;
    if (in) {
        if (done == nb) {
#pragma unroll
            for (int q = 0; q < NB; ++q)
                if (q >= NB - nb) T[r + (int64_t)(q - (NB - nb)) * S] = P[q];
        }
        used[r] = mine;
    }
    if (r < done) piv[k0 + r] = s_piv[r];
    // after a zero pivot the remaining columns keep an in-range row index so that the
    // update and extraction kernels stay in bounds (the error flag is already set)
    if (r >= done && r < nb) piv[k0 + r] = 0;
}

// Update of the columns [c0, c1) outside the panel [k0, k0+nb): t <- t + E t[piv] for TW
// columns per CTA (blockIdx.x) of odd block blockIdx.y, shift blockIdx.z; a column t left of
// the panel is a finished column of the inverse, one right of it is still to be eliminated.
// The CTA owns its columns whole (their pivot rows are read before they are replaced)
// and walks the rows in chunks of 128: a thread holds 4 rows x TW / 8 columns, so that
// one step of the sum costs 4 + TW / 8 shared-memory loads for TW / 2 complex products
// and FP32 arithmetic, not shared memory, is the bound (complex128: the FP64 pipe).
// The last chunk computes only the 32-row groups that it has (S = 400 has 13 of 16: one
// solve of the 240k-unknown shell 40.7 -> 39.1 ms).  Packed FP32 pairs instead of single
// multiply-adds were slower (72k-unknown shell, 16 shifts: 16.7 ms in this kernel against 13.6),
// as the pivot rows then take twice the shared-memory reads.
constexpr int kUpdRows = 128;

// NI groups of 32 rows from r0 on: the sums of the panel's columns, added and stored
template <typename C, int NB, int TW, int NI, typename Column>
__device__ __forceinline__ void update_rows(const C *src, C *T, const C (*es)[kUpdRows], const C (*tp)[TW],
                                            const int *used, int S, int r0, int k0, int nb, int nt, Column column) {
    constexpr int CT = TW / 8;   // columns per thread
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    C acc[NI][CT];
#pragma unroll
    for (int i = 0; i < NI; ++i) {
        const int r = r0 + tx + 32 * i;
        // a pivot row of the panel starts from zero
        const bool keep = r < S && !(used[r] > k0 && used[r] <= k0 + nb);
#pragma unroll
        for (int t = 0; t < CT; ++t)
            acc[i][t] = (keep && ty * CT + t < nt) ? src[r + (int64_t)column(ty * CT + t) * S] : czero<C>();
    }
    __syncthreads();
#pragma unroll 4
    for (int c = 0; c < NB; ++c) {
        C e[NI], t4[CT];
#pragma unroll
        for (int i = 0; i < NI; ++i) e[i] = es[c][tx + 32 * i];
#pragma unroll
        for (int t = 0; t < CT; ++t) t4[t] = tp[c][ty * CT + t];
#pragma unroll
        for (int i = 0; i < NI; ++i)
#pragma unroll
            for (int t = 0; t < CT; ++t) acc[i][t] = cfma(acc[i][t], e[i], t4[t]);
    }
#pragma unroll
    for (int i = 0; i < NI; ++i) {
        const int r = r0 + tx + 32 * i;
#pragma unroll
        for (int t = 0; t < CT; ++t)
            if (r < S && ty * CT + t < nt) T[r + (int64_t)column(ty * CT + t) * S] = acc[i][t];
    }
}

template <typename C, int NB, int TW>
__global__ void __launch_bounds__(256) k_update(FV<C> v, int k0, int nb, int c0, int c1, int stride, int split) {
    __shared__ __align__(16) C tp[NB][TW];
    __shared__ __align__(16) C es[NB][kUpdRows];
    const int S = v.S;
    const int64_t o = blockIdx.y, sh = blockIdx.z;
    C *T = v.T + sh * v.t_stride + o * v.t_block;
    const C *src = k0 == 0 ? diag_block(v, o, sh, stride) : T;
    const int *piv = v.piv + sh * v.p_stride + o * S, *used = v.used + sh * v.p_stride + o * S;
    // columns of this CTA, counted from c0 without the panel's own
    after_previous();
    const int part = blockIdx.x % split;
    const int j0 = blockIdx.x / split * TW, nt = c1 - c0 - nb - j0;
    auto column = [&](int t) { const int j = c0 + j0 + t; return j < k0 ? j : j + nb; };
    for (int idx = threadIdx.x; idx < TW * NB; idx += 256) {
        const int c = idx % NB, t = idx / NB;
        tp[c][t] = (t < nt && c < nb) ? src[piv[k0 + c] + (int64_t)column(t) * S] : czero<C>();
    }
    if (split > 1)   // every CTA of the cluster has read the columns' pivot rows
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    const C *E = T + (int64_t)k0 * S;
    for (int r0 = part * kUpdRows; r0 < S; r0 += split * kUpdRows) {
        __syncthreads();
        for (int idx = threadIdx.x; idx < NB * kUpdRows; idx += 256) {
            const int rr = idx % kUpdRows, c = idx / kUpdRows;
            es[c][rr] = (r0 + rr < S && c < nb) ? E[r0 + rr + (int64_t)c * S] : czero<C>();
        }
        if (S - r0 > 96) update_rows<C, NB, TW, 4>(src, T, es, tp, used, S, r0, k0, nb, nt, column);
        else if (S - r0 > 64) update_rows<C, NB, TW, 3>(src, T, es, tp, used, S, r0, k0, nb, nt, column);
        else if (S - r0 > 32) update_rows<C, NB, TW, 2>(src, T, es, tp, used, S, r0, k0, nb, nt, column);
        else update_rows<C, NB, TW, 1>(src, T, es, tp, used, S, r0, k0, nb, nt, column);
    }
    before_next();
}

// The inverse from the reduced work matrix: row piv[k] of T is row k of the inverse and
// column k of T is its column piv[k] (column-major S x S, all shifts).
template <typename C>
__global__ void k_extract(FV<C> v, BcrLevel lv, int nodd, int top, int nshift) {
    const int S = v.S;
    const int64_t SS = (int64_t)S * S, pershift = (int64_t)nodd * SS, total = pershift * nshift;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t sh = idx / pershift;
        const int64_t ws = idx - sh * pershift;
        const int64_t o = ws / SS;
        const int64_t w = ws - o * SS;
        const int c = (int)(w / S), k = (int)(w - (int64_t)c * S);
        const C *T = v.T + sh * v.t_stride + o * v.t_block;
        const int *piv = v.piv + sh * v.p_stride + o * S;
        const int64_t j = top ? 0 : (2 * o + 1) * lv.stride;
        v.Dinv[sh * v.f_stride + j * SS + k + (int64_t)piv[c] * S] = T[piv[k] + (int64_t)c * S];
    }
}

// acc += a b; complex128 skips the products with a zero part of a (most couplings are
// real or imaginary, and every FP64 product costs its pipe slot; the sums are the same).
__device__ __forceinline__ float2 couple(float2 acc, float2 a, float2 b) { return cfma(acc, a, b); }
__device__ __forceinline__ double2 couple(double2 acc, double2 a, double2 b) {
    if (a.y == 0.0) return mk(fma(a.x, b.x, acc.x), fma(a.x, b.y, acc.y));
    if (a.x == 0.0) return mk(fma(-a.y, b.y, acc.x), fma(a.y, b.x, acc.y));
    return cfma(acc, a, b);
}

// Level 0 update of the even blocks with their sparse couplings:
//   Dw_i -= rs (L_i H_jl + U_i G_jr),  L'_i = -rs L_i G_jl,  U'_i = -rs U_i H_jr.
// CTA = (chunk of CW columns, even index e, shift); one thread per row, which reads its
// row's coupling entries once, as padded rows (the level-0 rows of the sweep, with the row
// scale folded in), and accumulates the CW columns in registers.  The CW columns of the
// four matrices are staged in shared memory: an entry (about 30 per row) costs 2 CW reads
// of them, which gathered from L2 took 14.0 ms for 16 shifts of the 72k-unknown shell in
// complex64.  What was left was the wait for the entries, 15 of 20 stalled warps: loaded one
// batch ahead they took it from 7.3 to 4.1 ms (complex128 is bound by the FP64 pipe, and
// deeper batches only cost it registers: four shifts 8.5 ms with 1, 9.4 with 4).
template <typename C, int CW>
__global__ void __launch_bounds__(512) k_even_l0(FV<C> v, BcrLevel lv) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *sm = reinterpret_cast<C *>(smem_raw);   // [left H | left G | right G | right H], CW x S each
    const int S = v.S;
    const int64_t SS = (int64_t)S * S;
    const int64_t e = blockIdx.y, sh = blockIdx.z;
    const int64_t q = 2 * e;                 // position = original block at level 0
    const bool hasl = q >= 1, hasr = q + 1 < lv.Kl;
    const bool outl = (lv.lu_nL >= 0) && q >= 2, outr = (lv.lu_nU >= 0) && q + 2 < lv.Kl;
    const int c0 = blockIdx.x * CW;
    const int cn = min(CW, S - c0);
    const int ntile = (S + 31) / 32;
    C *Di = v.Dw + sh * v.f_stride + q * SS;
    const C *G = v.G + sh * v.f_stride, *H = v.H + sh * v.f_stride;
    {
        const int64_t off = (int64_t)c0 * S;
        const C *src[4] = {hasl ? H + (q - 1) * SS + off : nullptr, outl ? G + (q - 1) * SS + off : nullptr,
                           hasr ? G + (q + 1) * SS + off : nullptr, outr ? H + (q + 1) * SS + off : nullptr};
#pragma unroll
        for (int m = 0; m < 4; ++m)
            if (src[m])
                for (int i = threadIdx.x; i < cn * S; i += blockDim.x) sm[m * CW * S + i] = src[m][i];
    }
    __syncthreads();
    C *LU = v.LU + sh * v.lu_stride;
    const C *ev = v.ell_val + sh * v.ell_stride;
    const int first = (int)(q * S);   // padded slot of the block's first row
    for (int r = threadIdx.x; r < S; r += blockDim.x) {
        C dsum[CW], lsum[CW], usum[CW];
#pragma unroll
        for (int t = 0; t < CW; ++t) dsum[t] = lsum[t] = usum[t] = czero<C>();
        const int64_t ebase = ((q * ntile + r / 32) * (int64_t)v.ell_w) * 32 + (r & 31);
        // kAhead entries are loaded while the kAhead before them are summed (ell_w is a
        // multiple of 8)
        constexpr int kAhead = sizeof(C) == 8 ? 4 : 1;
        int ncol[kAhead];
        C na[kAhead];
        auto load = [&](int k) {
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                ncol[u] = k < v.ell_w ? v.ell_col[ebase + (int64_t)(k + u) * 32] : -1;
                if (k < v.ell_w) na[u] = ev[ebase + (int64_t)(k + u) * 32];
            }
        };
        auto sum = [&](int col, C a) {
            if (col < 0) return;
            if (col < first) {   // left neighbour j = q - 1
                const C *x = sm + (col - first + S);
#pragma unroll
                for (int t = 0; t < CW; ++t) {
                    dsum[t] = couple(dsum[t], a, x[t * S]);
                    if (outl) lsum[t] = couple(lsum[t], a, x[(CW + t) * S]);
                }
            } else {             // right neighbour j = q + 1
                const C *x = sm + 2 * CW * S + (col - first - S);
#pragma unroll
                for (int t = 0; t < CW; ++t) {
                    dsum[t] = couple(dsum[t], a, x[t * S]);
                    if (outr) usum[t] = couple(usum[t], a, x[(CW + t) * S]);
                }
            }
        };
        load(0);
        for (int k = 0; k < v.ell_w; k += kAhead) {
            int col[kAhead];
            C a[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                col[u] = ncol[u];
                a[u] = na[u];
            }
            load(k + kAhead);
#pragma unroll
            for (int u = 0; u < kAhead; ++u) sum(col[u], a[u]);
        }
#pragma unroll
        for (int t = 0; t < CW; ++t)
            if (t < cn) {
                const int64_t col = (int64_t)(c0 + t) * S;
                Di[r + col] = Di[r + col] - dsum[t];
                if (outl) LU[(lv.lu_nL + e) * SS + r + col] = -lsum[t];
                if (outr) LU[(lv.lu_nU + e) * SS + r + col] = -usum[t];
            }
    }
}

// Level 0: G_j = D_j^-1 (R L_j) and H_j = D_j^-1 (R U_j) from the couplings by column:
// column c of G_j = sum over the entries (k, e) of column c of L_j of rs_k a_e D_j^-1[:, k]
// (D_j^-1 is the inverse of the row-scaled block, so this is D^-1 L of the unscaled
// system).  CTA = (chunk of kGhCW columns, odd index o, shift): the entries of one column
// are staged in shared memory, then one thread per row accumulates.
constexpr int kGhCW = 8;
constexpr int kGhBuf = 512;
template <typename C>
__global__ void __launch_bounds__(512) k_gh_l0(FV<C> v) {
    __shared__ int sk[kGhBuf];
    __shared__ C sv[kGhBuf];
    const int S = v.S;
    const int64_t SS = (int64_t)S * S;
    const int64_t o = blockIdx.y, sh = blockIdx.z, j = 2 * o + 1;
    const int c0 = blockIdx.x * kGhCW, c1 = min(S, c0 + kGhCW);
    const C *Di = v.Dinv + sh * v.f_stride + j * SS;
    const double *rs = v.rscale + sh * v.np + j * S;
    for (int side = 0; side < 2; ++side) {
        const int *ptr = v.cc_ptr + (2 * o + side) * (int64_t)(S + 1);
        C *out = (side ? v.H : v.G) + sh * v.f_stride + j * SS;
        for (int c = c0; c < c1; ++c) {
            C acc[4] = {czero<C>(), czero<C>(), czero<C>(), czero<C>()};   // rows r, r + nt, ...
            for (int b0 = ptr[c]; b0 < ptr[c + 1]; b0 += kGhBuf) {
                const int nb = min(kGhBuf, ptr[c + 1] - b0);
                __syncthreads();
                for (int t = threadIdx.x; t < nb; t += blockDim.x) {
                    const int k = v.cc_row[b0 + t];
                    sk[t] = k;
                    sv[t] = from_c128<C>(rs[k] * v.aval[v.cc_src[b0 + t]]);
                }
                __syncthreads();
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const int r = threadIdx.x + h * blockDim.x;
                    if (r < S)
                        for (int t = 0; t < nb; ++t) acc[h] = cfma(acc[h], Di[r + (int64_t)sk[t] * S], sv[t]);
                }
            }
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                const int r = threadIdx.x + h * blockDim.x;
                if (r < S) out[r + (int64_t)c * S] = acc[h];
            }
        }
    }
}

unsigned grid_for(int64_t work, int threads, int num_sms) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>((work + threads - 1) / threads, 16LL * num_sms));
}

// Gauss-Jordan of the nodd work matrices T_o of every shift, then extraction.  Complex64:
// panels of NB columns, each followed by the update of all other columns.  Complex128, where
// that update would keep the FP64 pipe busy: the panels' updates stay within a group of
// kGroup columns, whose transform is then applied to the other columns as one product on
// the tensor cores (gemm_oz.cu), so that the FP64 pipe does kGroup / S of the work.  Wider
// groups leave more of it there, narrower ones make more products (four shifts of the
// 72k-unknown shell, S = 240, factorised and solved: 104.6, 99.8 and 107.6 ms for 32, 48 and
// 64; without groups 175 ms).
constexpr int kGroup = 48;
template <typename C, int NB, int MAXT>
int gauss_jordan(kore_plan *p, const FV<C> &v, const BcrLevel &lv, int nodd, int top, int nshift) {
    const int S = p->S;
    const int pthreads = ((S + 31) / 32) * 32;
    // A group's product has fixed costs of about 50 us (four launches, one tile's chain); the
    // FP64 products that it replaces, four multiply-adds each, run at two per SM and clock.  Per
    // shift, as the two forms round differently and a shift's factors must not depend on how
    // many others share the launches.  Limits of 200,000, 100,000, 50,000 and 20,000 cycles,
    // factorisation of 1, 4 and 8 shifts: 60 blocks of S = 96, 4.45, 6.1, 8.6 ms; 4.45, 6.0, 8.7;
    // 4.43, 5.6, 8.0; 4.64, 5.7, 7.5; 300 of S = 240, 35.2, 92.6, 172; 35.3, 91.6, 169; 35.7, 91.4,
    // 169; 36.8, 91.9, 168.  (With a right-hand side one shift of S = 96 takes 4.67 ms ungrouped,
    // 4.75 with level 0 grouped, which is at 87,000.)
    const int64_t fma = 4LL * nodd * S * std::max(0, S - kGroup) * kGroup;
    const int group = (sizeof(C) == 16 && fma / (2 * p->num_sms) > 90000) ? kGroup : S;
    for (int g0 = 0; g0 < S; g0 += group) {
        const int g1 = std::min(S, g0 + group);
        for (int k0 = g0; k0 < g1; k0 += NB) {
            const int nb = std::min(NB, g1 - k0), ncols = g1 - g0 - nb;
            KORE_TRY(kore_launch_chained(p->stream, k_panel<C, NB, MAXT>, dim3(nodd, nshift), panel_threads(pthreads), 1, v, k0, nb,
                                    lv.stride));
            if (ncols == 0) continue;
            // 32 columns per CTA re-read the panel least; levels with few blocks take 8, so
            // that their CTAs still cover the GPU, and share the row chunks among a cluster's
            // CTAs, as a chunk then is a chain of loads and a few products (two shifts of the MAC
            // shell, S = 360: 9.37 -> 9.31 ms; the 240k-unknown shell: 38.4 -> 38.2 ms)
            if ((int64_t)nodd * nshift * kore_div_up(ncols, 32) >= 2 * p->num_sms) {
                KORE_TRY(kore_launch_chained(p->stream, k_update<C, NB, 32>, dim3(kore_div_up(ncols, 32), nodd, nshift), 256, 1, v, k0, nb,
                                        g0, g1, lv.stride, 1));
            } else {
                const int split = (int)kore_div_up(S, kUpdRows);   // at most 8, a portable cluster
                KORE_TRY(kore_launch_chained(p->stream, k_update<C, NB, 8>, dim3(kore_div_up(ncols, 8) * split, nodd, nshift), 256,
                                        split, v, k0, nb, g0, g1, lv.stride, split));
            }
        }
        if (g1 - g0 < S) KORE_TRY(kore_group_update_oz(p, lv, nodd, g0, g1));
    }
    k_extract<C><<<grid_for((int64_t)nodd * S * S * nshift, 256, p->num_sms), 256, 0, p->stream>>>(v, lv, nodd, top,
                                                                                                nshift);
    KORE_LAUNCHED(1);
    KORE_CUDA_TRY(cudaGetLastError());
    return KORE_OK;
}

template <typename C, int NB, int MAXT>
int factor_levels(kore_plan *p) {
    const int S = p->S, K = p->K, ns = p->fw_n;
    const int64_t SS = (int64_t)S * S;
    cudaStream_t st = p->stream;
    const FV<C> v = make_fv<C>(p);
    // working diagonal blocks from the CSR
    k_Dw_init<C><<<grid_for((int64_t)K * SS * ns, 256, p->num_sms), 256, 0, st>>>(v, ns);
    k_Dw_scatter<C><<<grid_for(p->np * 32 * ns, 256, p->num_sms), 256, 0, st>>>(v, ns);
    KORE_LAUNCHED(2);
    for (int l = 0; l < p->nlev; ++l) {
        const BcrLevel &lv = p->lev[l];
        // D_j^-1 of the odd blocks by Gauss-Jordan
        KORE_TRY((gauss_jordan<C, NB, MAXT>(p, v, lv, lv.nodd, 0, ns)));
        const int th = std::min(512, ((S + 31) / 32) * 32);   // rows per pass (S <= 1024: two passes at most)
        if (l == 0) {
            // G_j, H_j from the sparse couplings (complex64: refined on the tensor cores),
            // then the even blocks
            k_gh_l0<C><<<dim3(kore_div_up(S, kGhCW), lv.nodd, ns), th, 0, st>>>(v);
            KORE_LAUNCHED(1);
            if (sizeof(C) == sizeof(float2)) KORE_TRY(kore_gh_update_tc(p, lv, 1));
            // columns per CTA: 4 while they leave room for two CTAs per SM in shared memory
            // (S = 800 in complex64: 102 KB), else 2.  8 took 97 registers in complex64, which
            // left too few warps to cover the entries' loads: 6.0 against 4.1 ms for 16 shifts
            // of the 72k-unknown shell, 2.7 against 1.7 ms for one of the 240k-unknown shell;
            // 2 took 5.3 and 2.2 ms.
            const size_t per = (size_t)4 * S * sizeof(C);
            const int cw = 4 * per <= 110 * 1024 ? 4 : 2;
            auto even = cw == 4 ? k_even_l0<C, 4> : k_even_l0<C, 2>;
            KORE_TRY(kore_allow_max_dyn_smem(even, p->device));
            even<<<dim3(kore_div_up(S, cw), lv.neven, ns), th, cw * per, st>>>(v, lv);
            KORE_LAUNCHED(1);
        } else if (sizeof(C) == sizeof(float2)) {
            // complex64: tensor cores (3xTF32)
            KORE_TRY(kore_gh_update_tc(p, lv, 0));
            KORE_TRY(kore_even_update_tc(p, lv));
        } else {
            // complex128: tensor cores (digits)
            KORE_TRY(kore_gh_update_oz(p, lv));
            KORE_TRY(kore_even_update_oz(p, lv));
        }
        KORE_CUDA_TRY(cudaGetLastError());
    }
    // the last active block (block 0); stride 0 maps odd index 0 to block 0
    BcrLevel top{};
    top.Kl = 1;
    top.stride = 0;
    top.lu_L = top.lu_U = top.lu_nL = top.lu_nU = -1;
    KORE_TRY((gauss_jordan<C, NB, MAXT>(p, v, top, 1, 1, ns)));
    return KORE_OK;
}

// A panel row lives in one thread's registers: NB complex values.  512 threads leave 128
// registers each (NB = 32 complex64, 16 complex128), 1024 leave 64.
template <typename C>
int factor_dispatch(kore_plan *p) {
    constexpr int NB = sizeof(C) == 8 ? 32 : 16;
    if (p->S <= 256) return factor_levels<C, NB, 256>(p);
    if (p->S <= 512) return factor_levels<C, NB, 512>(p);
    return factor_levels<C, NB / 2, 1024>(p);
}

}  // namespace

// Level table of the reduction for K blocks.
void kore_build_levels(kore_plan *p) {
    p->lev.clear();
    std::vector<int> Ks;
    for (int Kl = p->K; Kl > 1; Kl = Kl - Kl / 2) Ks.push_back(Kl);
    p->nlev = (int)Ks.size();
    p->nodd_max = 1;
    int64_t lu = 0;
    std::vector<int64_t> offL(p->nlev + 1, -1), offU(p->nlev + 1, -1);
    for (int l = 1; l < p->nlev; ++l) {
        offL[l] = lu;
        lu += Ks[l];
        offU[l] = lu;
        lu += Ks[l];
    }
    int stride = 1;
    for (int l = 0; l < p->nlev; ++l) {
        BcrLevel lv;
        lv.Kl = Ks[l];
        lv.stride = stride;
        lv.nodd = Ks[l] / 2;
        lv.neven = Ks[l] - lv.nodd;
        lv.lu_L = offL[l];
        lv.lu_U = offU[l];
        lv.lu_nL = (l + 1 < p->nlev) ? offL[l + 1] : -1;
        lv.lu_nU = (l + 1 < p->nlev) ? offU[l + 1] : -1;
        p->lev.push_back(lv);
        p->nodd_max = std::max(p->nodd_max, lv.nodd);
        stride *= 2;
    }
    p->lu_mats = std::max<int64_t>(lu, 1);
}

namespace {

// (Re)allocate the per-shift buffers for `cap` shifts of elements of `elt` bytes.
int ensure_factor_storage(kore_plan *p, int cap, size_t elt) {
    if (p->factor_elt == elt && p->shift_cap >= cap) return KORE_OK;
    void **bufs[] = {&p->d_Dinv, &p->d_Gm, &p->d_Hm, &p->d_Dw, &p->d_LU, &p->d_T, &p->d_sweep,
                     (void **)&p->d_rscale, (void **)&p->d_piv, (void **)&p->d_used,
                     (void **)&p->d_sigma, (void **)&p->d_minf, (void **)&p->d_bb, (void **)&p->d_xb, (void **)&p->d_rb,
                     (void **)&p->d_bn, (void **)&p->d_rn, (void **)&p->d_part, (void **)&p->d_ir, (void **)&p->d_tick,
                     &p->d_ell_val, &p->d_tctab, &p->d_oz};
    for (void **b : bufs) {
        if (*b) cudaFree(*b);
        *b = nullptr;
    }
    p->bytes -= p->factor_bytes;
    p->factor_bytes = 0;
    p->factor_elt = 0;
    p->shift_cap = 0;
    p->oz_bytes = 0;
    const size_t before = p->bytes;
    const size_t c = (size_t)cap;
    KORE_TRY(kore_alloc(p, &p->d_Dinv, c * p->f_stride() * elt));
    KORE_TRY(kore_alloc(p, &p->d_Gm, c * p->f_stride() * elt));
    KORE_TRY(kore_alloc(p, &p->d_Hm, c * p->f_stride() * elt));
    KORE_TRY(kore_alloc(p, &p->d_Dw, c * p->f_stride() * elt));
    KORE_TRY(kore_alloc(p, &p->d_LU, c * p->lu_stride() * elt));
    KORE_TRY(kore_alloc(p, &p->d_T, c * p->nodd_max * p->t_block(elt) * elt));
    KORE_TRY(kore_alloc(p, &p->d_sweep, c * p->sweep_vec_elems() * elt));
    KORE_TRY(kore_alloc(p, (void **)&p->d_rscale, c * p->np * sizeof(double)));
    KORE_TRY(kore_alloc(p, (void **)&p->d_piv, c * p->p_stride() * sizeof(int)));
    KORE_TRY(kore_alloc(p, (void **)&p->d_used, c * p->p_stride() * sizeof(int)));
    KORE_TRY(kore_alloc(p, (void **)&p->d_sigma, c * sizeof(double2)));
    KORE_TRY(kore_alloc(p, (void **)&p->d_minf, c * sizeof(double)));
    KORE_TRY(kore_alloc(p, (void **)&p->d_bb, c * p->np * sizeof(double2)));
    KORE_TRY(kore_alloc(p, (void **)&p->d_xb, c * p->np * sizeof(double2)));
    KORE_TRY(kore_alloc(p, (void **)&p->d_rb, c * p->np * sizeof(double2)));
    KORE_TRY(kore_alloc(p, (void **)&p->d_bn, c * sizeof(double)));
    KORE_TRY(kore_alloc(p, (void **)&p->d_rn, c * sizeof(double)));
    // per-CTA maxima of the residual products: (np / 64 + np / 8 + 2) CTAs at most, 2 each
    KORE_TRY(kore_alloc(p, (void **)&p->d_part, c * 2 * (size_t)(p->np / 64 + p->np / 8 + 1024) * sizeof(double)));
    KORE_TRY(kore_alloc(p, (void **)&p->d_ir, c * sizeof(IrState)));
    KORE_TRY(kore_alloc(p, &p->d_ell_val, c * std::max<int64_t>(p->ell_stride(), 1) * elt));
    if (elt == sizeof(float2)) KORE_TRY(kore_alloc(p, &p->d_tctab, (size_t)kore_tc_table_bytes(p, cap)));
    else {
        const int64_t oz = kore_oz_workspace_bytes(p->S, p->K, cap);
        KORE_TRY(kore_alloc(p, &p->d_oz, (size_t)oz));
        p->oz_bytes = oz;
    }
    KORE_CUDA_TRY(cudaMemset(p->d_LU, 0, c * p->lu_stride() * elt));
    KORE_CUDA_TRY(cudaMemset(p->d_piv, 0, c * p->p_stride() * sizeof(int)));
    KORE_CUDA_TRY(cudaMemset(p->d_used, 0, c * p->p_stride() * sizeof(int)));
    KORE_CUDA_TRY(cudaMemset(p->d_ir, 0, c * sizeof(IrState)));
    KORE_TRY(kore_alloc(p, (void **)&p->d_tick, c * sizeof(unsigned)));
    KORE_CUDA_TRY(cudaMemset(p->d_tick, 0, c * sizeof(unsigned)));
    p->sweep_launch.reset();
    p->factor_bytes = p->bytes - before;
    p->factor_elt = elt;
    p->shift_cap = cap;
    return KORE_OK;
}

}  // namespace

namespace {

// Row scales, norms and level-0 couplings of the factor window, then its levels.
template <typename C>
int factor_window(kore_plan *p) {
    const int lo = p->fw_lo, ns = p->fw_n;
    const unsigned grid = kore_div_up(p->np, 256);
    double *red = p->d_part;   // scratch: grid x ns doubles fit the residual partials buffer
    k_rowinfo<C><<<grid, 256, 0, p->stream>>>(make_fv<C>(p), ns, red);
    k_minf<<<ns, 256, 0, p->stream>>>(red, (int)grid, p->d_minf + lo);
    KORE_LAUNCHED(2);
    if (p->ell_stride() > 0) {
        k_ell_fill<C><<<dim3(std::min<unsigned>(kore_div_up(p->ell_stride(), 256), 4096u), ns), 256, 0, p->stream>>>(
            p->ell_stride(), p->ell_w, (p->S + 31) / 32, p->S, p->np, p->d_ell_src, p->d_aval,
            p->d_rscale + (int64_t)lo * p->np, static_cast<C *>(p->d_ell_val) + (int64_t)lo * p->ell_stride());
        KORE_LAUNCHED(1);
    }
    return factor_dispatch<C>(p);
}

// Factorises the factor window; the norms of its shifts come back with the one wait at the end.
int run_window(kore_plan *p) {
    if (p->prof) KORE_TRY(kore_prof_mark(p, 1, true));
    KORE_TRY(p->prec == KORE_PREC_FP64 ? factor_window<double2>(p) : factor_window<float2>(p));
    if (p->prof) KORE_TRY(kore_prof_mark(p, 1, false));
    KORE_CUDA_TRY(cudaMemcpyAsync(p->minfs.data() + p->fw_lo, p->d_minf + p->fw_lo, p->fw_n * sizeof(double),
                                  cudaMemcpyDeviceToHost, p->stream));
    KORE_CUDA_TRY(cudaStreamSynchronize(p->stream));
    p->minf = p->minfs[0];
    return kore_check_device_error(p);
}

}  // namespace

int kore_factor_impl(kore_plan *p, int nshift, const double *sigmas, int precision) {
    if (precision != KORE_PREC_FP64 && precision != KORE_PREC_MIXED) return KORE_EINVAL;
    if (nshift <= 0 || !sigmas) return KORE_EINVAL;
    const size_t elt = (precision == KORE_PREC_FP64) ? sizeof(double2) : sizeof(float2);
    p->factored = false;
    KORE_TRY(ensure_factor_storage(p, nshift, elt));
    p->prec = precision;
    p->nshift = nshift;
    p->fw_lo = 0;
    p->fw_n = nshift;
    p->sigmas.assign(nshift, mk(0.0, 0.0));
    p->minfs.assign(nshift, 0.0);
    for (int s = 0; s < nshift; ++s) p->sigmas[s] = mk(sigmas[2 * s], sigmas[2 * s + 1]);
    p->sigma_re = sigmas[0];
    p->sigma_im = sigmas[1];
    KORE_CUDA_TRY(cudaMemcpyAsync(p->d_sigma, p->sigmas.data(), nshift * sizeof(double2), cudaMemcpyHostToDevice,
                                  p->stream));
    KORE_TRY(run_window(p));
    p->factored = true;
    return KORE_OK;
}

// Re-factorise one shift of a factorised plan: shift `slot` becomes A - sigma B and the
// other shifts keep their factors (the factor window is narrowed to the slot for the
// launches).  A batched eigensolve uses it to start a new target in a slot whose target
// has finished while the other slots carry on.
int kore_factor_slot(kore_plan *p, int slot, double sigma_re, double sigma_im) {
    if (!p->factored || slot < 0 || slot >= p->nshift) return KORE_EINVAL;
    p->factored = false;
    p->sigmas[slot] = mk(sigma_re, sigma_im);
    if (slot == 0) { p->sigma_re = sigma_re; p->sigma_im = sigma_im; }
    KORE_CUDA_TRY(cudaMemcpyAsync(p->d_sigma + slot, &p->sigmas[slot], sizeof(double2), cudaMemcpyHostToDevice,
                                  p->stream));
    p->fw_lo = slot;
    p->fw_n = 1;
    const int s = run_window(p);
    p->fw_lo = 0;
    p->fw_n = p->nshift;
    if (s != KORE_OK) return s;
    p->factored = true;
    return KORE_OK;
}

int kore_factor_reserve(kore_plan *p, int nslot, int precision) {
    if (nslot <= 0 || (precision != KORE_PREC_FP64 && precision != KORE_PREC_MIXED)) return KORE_EINVAL;
    const size_t elt = (precision == KORE_PREC_FP64) ? sizeof(double2) : sizeof(float2);
    p->factored = false;
    KORE_TRY(ensure_factor_storage(p, nslot, elt));
    p->prec = precision;
    p->nshift = nslot;
    p->fw_lo = 0;
    p->fw_n = nslot;
    // no slot holds a shift yet (NaN matches no target)
    p->sigmas.assign(nslot, mk(NAN, NAN));
    p->minfs.assign(nslot, 0.0);
    p->sigma_re = p->sigma_im = NAN;
    KORE_CUDA_TRY(cudaMemcpyAsync(p->d_sigma, p->sigmas.data(), nslot * sizeof(double2), cudaMemcpyHostToDevice,
                                  p->stream));
    KORE_CUDA_TRY(cudaMemcpyAsync(p->d_minf, p->minfs.data(), nslot * sizeof(double), cudaMemcpyHostToDevice,
                                  p->stream));
    KORE_CUDA_TRY(cudaStreamSynchronize(p->stream));
    p->factored = true;   // slot by slot from here (kore_factor_slot)
    return KORE_OK;
}
