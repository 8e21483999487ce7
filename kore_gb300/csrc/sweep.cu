// Solves with the block-cyclic-reduction factors of factor.cu, sparse products and
// the FP64 refinement loop.
//
// (A - sigma B) x = b with row scaling R and s = ||b||_inf (keeps complex64 in range):
// the right-hand side c = s^-1 R b is reduced level by level exactly as the blocks were,
//     level l, odd blocks j:   z_j = D_j^-1 f_j
//     level l, even blocks i:  f_i <- f_i - L_i z_jl - U_i z_jr        (CSR couplings at level 0)
// the last block is solved, x_0 = D_0^-1 f_0, and the levels are unwound in reverse,
//     level l >= 1, odd blocks j:   x_j = z_j - G_j x_jl - H_j x_jr,
//     level 0, odd blocks j:        g_j = c_j - L_j x_{j-1} - U_j x_{j+1},  x_j = D_j^-1 g_j
// then x <- s x.  At level 0 the couplings are sparse, so forming g_j from them and
// multiplying by D_j^-1 reads one dense block instead of the two of G_j, H_j.  One cooperative
// persistent kernel runs all phases (about 3 log2 K of them) as a dataflow over tiles of 32
// (or 8) rows: a tile starts as soon as the entries it reads are there (each entry shows its
// own readiness), and the factor blocks stream from HBM through shared memory by TMA.
//
// Every kernel here works on all factorised shifts at once (shift s: its own factors,
// row scales and vectors at offset s * stride), so a batch of forcing frequencies is
// one sweep launch.
//
// In mixed precision the factors are complex64 and the result is refined in FP64:
//     r = b - (A - sigma B) x,  x += M32^-1 r   until ||r||_inf <= tol (||M||_inf ||x||_inf + ||b||_inf).
#include "kore_internal.cuh"
#include "kore_tma.cuh"
#include <cstddef>
#include <cstring>
#include <memory>
#include <map>
#include <mutex>
#include <tuple>

namespace {

__device__ __forceinline__ double2 ldg(const double2 *p) { return __ldg(p); }
__device__ __forceinline__ float2 ldg(const float2 *p) { return __ldg(p); }
template <typename C> __device__ __forceinline__ C shfl_xor(C v, int o) {
    v.x = __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y = __shfl_xor_sync(0xffffffffu, v.y, o);
    return v;
}

struct SweepArgs {
    int K, S, nlev, nshift;
    const BcrLevel *levs;
    const void *Dinv, *G, *H, *LU;
    int64_t f_stride, lu_stride;     // per-shift strides of the factor blocks (elements)
    const int *ell_col;              // level-0 couplings as padded rows (kore_plan::d_ell_*)
    const void *ell_val;
    int ell_w;
    int64_t ell_stride;              // per-shift stride of ell_val (elements)
    const double2 *b;                // nshift x np right-hand sides (complex128, padded)
    const double *rscale;            // nshift x np
    const double *bnorm;             // nshift scalings
    void *vecs;                      // per shift the sweep's vectors (sweep_vec_elems), all bits set
                                     // before the launch
    int64_t vec_stride;
    double2 *out;                    // nshift x np
    int accumulate;
    int *err;
    const int *skip;                 // shift s is skipped when skip[s * skip_stride] != 0
    int skip_stride;
    unsigned live_mask;              // shift s (< 32) takes part only when bit s is set
    int *count;                      // sweeps that ran
    int *count_total;
};

constexpr int kMaxLevels = 24;

// bit s of a live-shift mask (shifts past 31 always take part)
__host__ __device__ __forceinline__ bool mask_has(unsigned mask, int64_t s) {
    return s >= 32 || ((mask >> s) & 1u);
}

// An entry of the sweep's vectors is written once per sweep.  Before the sweep all its bits
// are set, a NaN that is never stored, so a reader sees by the entry itself whether
// it is there: no counter, fence or flag stands between a tile's result and its use.
// (FP32 arithmetic gives one NaN of other bits.  FP64 addition and multiplication keep the bits
// of a NaN operand, so one of all bits set could come from a caller's vector: it is stored as
// another NaN.)  The 8
// bytes of a complex64 entry and each half of a complex128 one are written and read as one
// access (relaxed, at L2), and a complex128 entry is there when both halves are.
__device__ __forceinline__ void st_entry(float2 *p, float2 v) {
    const unsigned long long b = (unsigned long long)__float_as_uint(v.x) | ((unsigned long long)__float_as_uint(v.y) << 32);
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(b) : "memory");
}
__device__ __forceinline__ double not_the_mark(double v) {
    return __double_as_longlong(v) == -1ll ? __longlong_as_double(0x7ff8000000000000ll) : v;
}
__device__ __forceinline__ void st_entry(double2 *p, double2 v) {
    v = mk(not_the_mark(v.x), not_the_mark(v.y));
    asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(v.x), "d"(v.y) : "memory");
}
__device__ __forceinline__ float2 ld_entry(const float2 *p) {
    unsigned long long b;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(b) : "l"(p) : "memory");
    return make_float2(__uint_as_float((unsigned)b), __uint_as_float((unsigned)(b >> 32)));
}
__device__ __forceinline__ double2 ld_entry(const double2 *p) {
    double2 v;
    asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ bool unset(float2 v) { return __float_as_uint(v.x) == 0xffffffffu; }
__device__ __forceinline__ bool unset(double2 v) {
    return __double_as_longlong(v.x) == -1ll || __double_as_longlong(v.y) == -1ll;
}

// Iteration limit of a wait for an entry (about a microsecond each): seconds.
constexpr unsigned kEntryLimit = 1u << 22;

// Reads (bounded) an entry until it is there; on timeout or an earlier error the error flag
// is set and the caller goes on (its result is then wrong, but the kernel ends).
template <typename C>
__device__ __noinline__ C wait_entry_long(const C *p, int *err) {
    C v = ld_entry(p);
    for (unsigned spins = 0; unset(v); v = ld_entry(p)) {
        if (ld_relaxed_i32(err) != 0) break;
        if (++spins > kEntryLimit) { atomicCAS(err, 0, KORE_DEVERR_FLAG); break; }
        __nanosleep(64);
    }
    return v;
}
template <typename C>
__device__ __forceinline__ C wait_entry(const C *p, int *err) {
    C v = ld_entry(p);
    for (int spins = 0; unset(v) && spins < 16; ++spins) v = ld_entry(p);
    return unset(v) ? wait_entry_long(p, err) : v;
}

// ----------------------------------------------------------------------------- the sweep kernel
// The tiles (32 rows of one block) of all stages are numbered in a topological order
//     A_0, B_0, A_1, B_1, ..., A_{L-1}, B_{L-1}, top, C_{L-1}, ..., C_1, E_0, C_0
// (A: z_j = D_j^-1 f_j, B: f_i -= L_i z_jl + U_i z_jr, C: x_j = z_j - G_j x_jl - H_j x_jr
// at levels >= 1; E_0: g_j = c_j - L_j x_jl - U_j x_jr and C_0: x_j = D_j^-1 g_j)
// and CTA c takes tiles c, c + G, c + 2G, ...  A tile waits for the entries it reads, each
// written by a tile of a lower number (st_entry, wait_entry).  Tiles are taken in increasing
// order by co-resident CTAs, so every wait is on a tile that some CTA is processing or has
// processed: no deadlock, and adjacent stages overlap.  Per shift there are four vectors: z
// and x (a block of each is written once), g (E_0), and f, which every level has its own copy
// of (level l's active blocks, l >= 1; level 0's is the right-hand side), so that every entry
// is written once.
//
// With completion counters (a fence and an atomic per tile, a checker warp that polled them
// and told the consumers, then the loads) a stage of the chain spent 2.9 us of its 4 us between
// one tile's result and the next tile's inputs.
//
// A tile of A, C, top or B at levels >= 1 reads one or two S x S blocks (stored
// column-major); they are cut into chunks of 32 rows x kCols columns (16 KB) that one
// producer thread copies with cp.async.bulk.tensor into a ring of shared-memory slots,
// each slot guarded by a "full" mbarrier (completed by the copy) and an "empty"
// mbarrier (one arrival per consumer warp).  The producer runs ahead through the CTA's
// tile sequence: the factor data of later tiles does not depend on the sweep, so it is
// fetched while the consumer warps wait for their input vectors.  B_0 and E_0 read the level-0
// couplings as padded rows (at most a few dozen entries per row) with plain coalesced loads
// instead.
constexpr int kTmaConsumerWarps = 4;
constexpr int kTmaConsumers = 32 * kTmaConsumerWarps;
// Variants: 2, 3 or 4 CTAs per SM (deeper rings per CTA, or more CTAs whose per-tile
// work -- input vectors, reduction, signalling -- overlaps the others' streaming) and
// chunks of 8 or 16 KB (the ring holds the same bytes; with smaller chunks a consumed
// chunk frees its slot sooner, so more of the ring is in flight).  The autotuner below
// picks one per plan shape; untuned sweeps use 4 CTAs per SM and 8 KB chunks.
struct TmaVariant { int cps, chunk; };
constexpr TmaVariant kTmaVariants[] = {{2, 16384}, {3, 16384}, {4, 16384}, {2, 8192}, {3, 8192}, {4, 8192}};
constexpr TmaVariant kTmaDefault = {4, 8192};
constexpr int kTmaThreads = kTmaConsumers + 32;   // + one producer warp
constexpr int kTileRows = 32;
// Stages with few tiles take tiles of 8 rows instead: a chunk then holds four times the
// columns and four times as many SMs work on the stage.  These stages are the chain of the
// upper levels, where a tile's own time counts.  complex128: its products (10.5 us per matrix
// of S = 240 on the FP64 pipe of one SM), so a warp's lanes share each row four ways (lane =
// row + 8 x column mod 4), with the four sums that a lane of a 32-row tile keeps.  complex64:
// its chunks' waits (2.8 us per matrix at S = 400; a quarter of the chunks, 0.7 us); a warp
// keeps its columns and their order.  The sums of both heights are the same bit for bit, as the
// height depends on the number of shifts (sweep_low_tiles).
constexpr int kLowRows = 8;
constexpr int kMaxRing = 24;
constexpr int kEllReg = 4;   // level-0 coupling entries per thread held in registers (width 32)
// input-vector loads in flight per consumer lane: a two-matrix tile's slice (about 2 S / 4
// entries per warp: 2 x 7 x 16 at S = 400 with 16 KB chunks, 2 x 13 x 8 with 8 KB) takes
// one round of L2 latency with 8, two with 4; the variants whose register budget
// (65536 / (160 CPS)) cannot hold 8 keep 4
template <typename C, int CPS> constexpr int fill_of() { return (CPS == 2 || (CPS == 3 && sizeof(C) == 8)) ? 8 : 4; }

enum { kMapDinv = 0, kMapG = 1, kMapH = 2, kMapLU = 3 };

struct SweepTmaParams {
    CUtensorMap maps[8];   // Dinv, G, H, LU: (2S reals, S columns, blocks, shifts), boxes of 32
                           // rows, then the same with boxes of 8
    int low_tiles;         // a stage with at most this many 32-row tiles takes 8-row tiles
    SweepArgs a;
    int nst;               // ring slots
};

template <typename C, int CHUNK> struct TmaShape {
    static constexpr int kCols = CHUNK / (kTileRows * (int)sizeof(C));   // columns per chunk
};

// One tile of the sweep: stage kind (0 A, 1 B, 2 top, 3 C, 4 E_0), level, shift, block
// of its rows, first row, the blocks it multiplies (map, block index within the map), and
// the blocks of its vectors, as element offsets into the shift's vectors.
struct TileJob {
    int kind, l, nmat, r0;
    bool low;            // 8 rows instead of 32
    bool from_b;         // its input vector is the right-hand side
    int64_t s, blk;
    int map[2];
    int64_t mblk[2];
    int64_t in[2];       // the vector each matrix multiplies (E_0, B_0: in[0] the vector gathered from)
    int64_t add;         // what the product is subtracted from (-1: nothing or the right-hand side)
    int64_t out;
};

// Shapes that decode_tile needs, in shared memory.
struct SweepShape {
    int S, L, K;
    BcrLevel lv[kMaxLevels];
    int64_t begin[3 * kMaxLevels + 3];   // first tile of each stage
    int tiles[3 * kMaxLevels + 2];       // tiles per block of each stage
    int64_t fo[kMaxLevels + 1];          // element offset of level l's f (l >= 1)
    int64_t x, g;                        // element offsets of x and g (z: 0)
};

__device__ __forceinline__ void decode_tile(int64_t n, int &k, const SweepShape &h, TileJob &t) {
    while (n >= h.begin[k + 1]) ++k;
    const int L = h.L, ntile = h.tiles[k];
    const int64_t S = h.S, loc = n - h.begin[k];
    if (k < 2 * L) { t.kind = (k & 1) ? 1 : 0; t.l = k >> 1; }
    else if (k == 2 * L) { t.kind = 2; t.l = L; }
    else if (k < 3 * L) { t.kind = 3; t.l = 3 * L - k; }
    else if (k == 3 * L) { t.kind = 4; t.l = 0; }
    else { t.kind = 3; t.l = 0; }
    const int nblk = (t.kind == 1) ? h.lv[t.l].neven : (t.kind == 2 ? 1 : h.lv[t.l].nodd);
    t.s = loc / ((int64_t)nblk * ntile);
    const int64_t rem = loc - t.s * nblk * ntile;
    const int64_t bi = rem / ntile;
    t.low = ntile > (S + kTileRows - 1) / kTileRows;
    t.r0 = (int)(rem - bi * ntile) * (t.low ? kLowRows : kTileRows);
    t.nmat = 1;
    t.from_b = false;
    t.add = -1;
    if (t.kind == 0) {
        const int64_t q = 2 * bi + 1, j = q * h.lv[t.l].stride;
        t.blk = j;
        t.map[0] = kMapDinv; t.mblk[0] = j;
        t.from_b = t.l == 0;
        t.in[0] = t.l == 0 ? 0 : h.fo[t.l] + q * S;
        t.out = j * S;
    } else if (t.kind == 1) {
        const BcrLevel lv = h.lv[t.l];
        const int64_t q = 2 * bi;
        t.blk = q * lv.stride;
        t.out = h.fo[t.l + 1] + bi * S;
        if (t.l > 0) {
            // L_q z_jl first when it exists, then U_q z_jr
            const bool hasl = q >= 1, hasr = q + 1 < lv.Kl;
            const int64_t jl = (q - 1) * lv.stride, jr = (q + 1) * lv.stride;
            t.map[0] = t.map[1] = kMapLU;
            t.mblk[0] = hasl ? lv.lu_L + q : lv.lu_U + q;
            t.in[0] = (hasl ? jl : jr) * S;
            t.mblk[1] = lv.lu_U + q;
            t.in[1] = jr * S;
            t.nmat = (int)hasl + (int)hasr;
            t.add = h.fo[t.l] + q * S;
        } else {
            t.nmat = 0;
            t.in[0] = 0;   // z
        }
    } else if (t.kind == 2) {
        t.blk = 0;
        t.map[0] = kMapDinv; t.mblk[0] = 0;
        t.from_b = L == 0;
        t.in[0] = L == 0 ? 0 : h.fo[L];
        t.out = h.x;
    } else if (t.kind == 3 && t.l > 0) {
        const BcrLevel lv = h.lv[t.l];
        const int64_t q = 2 * bi + 1, j = q * lv.stride;
        t.blk = j;
        t.map[0] = kMapG; t.mblk[0] = j; t.in[0] = h.x + (j - lv.stride) * S;
        if (q + 1 < lv.Kl) { t.map[1] = kMapH; t.mblk[1] = j; t.in[1] = h.x + (j + lv.stride) * S; t.nmat = 2; }
        t.add = j * S;
        t.out = h.x + j * S;
    } else if (t.kind == 3) {
        // C_0: x_j = D_j^-1 g_j
        const int64_t j = 2 * bi + 1;
        t.blk = j;
        t.map[0] = kMapDinv; t.mblk[0] = j; t.in[0] = h.g + j * S;
        t.out = h.x + j * S;
    } else {
        // E_0: g_j = c_j - L_j x_{j-1} - U_j x_{j+1} from the padded coupling rows
        t.blk = 2 * bi + 1;
        t.nmat = 0;
        t.in[0] = h.x;
        t.out = h.g + t.blk * S;
    }
}

template <typename C, int CPS, int CHUNK>
__global__ void __launch_bounds__(kTmaThreads, CPS) k_sweep_tma(const __grid_constant__ SweepTmaParams P) {
    using Shape = TmaShape<C, CHUNK>;
    constexpr int kCols = Shape::kCols;
    constexpr int kFill = fill_of<C, CPS>();
    constexpr bool kSplit = sizeof(C) == 16;   // low tiles: lanes share a row
    // Columns of a warp: runs of kRun, 4 kRun apart, the same in every variant, so that a sweep's
    // sums do not depend on the autotuner's choice (complex64: with 8 KB chunks of 32 rows a warp
    // then works on every other chunk).  complex128 keeps a sum for each of the run's four
    // columns, as low tiles have them on four lanes: the sums then depend neither on the height
    // of the tiles nor with it on the number of shifts.
    constexpr int kRun = sizeof(C) == 8 ? 16 : 4;
    constexpr bool kHalf = kCols < 4 * kRun;
    constexpr int kAcc = kSplit ? 4 : 1;
    const SweepArgs &a = P.a;
    const int nst = P.nst;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const int S = a.S, ns = a.nshift, L = a.nlev, K = a.K;
    const int nvec = (S + 4 * kCols - 1) / (4 * kCols) * (4 * kCols);   // whole chunks of either height
    unsigned char *ring = smem_raw;
    uint64_t *full = reinterpret_cast<uint64_t *>(smem_raw + (size_t)nst * CHUNK);
    uint64_t *empty = full + nst;
    C *vbuf = reinterpret_cast<C *>(empty + nst);   // 2 x nvec input vectors (each warp fills its columns)
    __shared__ C red[2][kTmaConsumerWarps][33];   // per-warp partial sums, by tile parity
    __shared__ SweepShape h;
    {
        bool all = true;
        for (int s = 0; s < ns; ++s)
            all = all && (!mask_has(a.live_mask, s) || (a.skip && a.skip[s * a.skip_stride] != 0));
        if (all) return;
    }
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (a.count && blockIdx.x == 0 && tid == 0) { atomicAdd(a.count, 1); atomicAdd(a.count_total, 1); }
    const int64_t np = (int64_t)K * S;
    const int ntile = (S + kTileRows - 1) / kTileRows;
    const int nstage = L > 0 ? 3 * L + 2 : 1;
    if (tid < L) h.lv[tid] = a.levs[tid];
    if (tid == 0) {
        for (int i = 0; i < nst; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], kTmaConsumerWarps); }
        mbar_fence_init();
    }
    if (tid == kTmaConsumers) for (int i = 0; i < 8; ++i) tma_prefetch_desc(&P.maps[i]);
    __syncthreads();
    if (tid == 0) {
        h.S = S; h.L = L; h.K = K;
        h.x = np;
        h.g = 2 * np;
        int64_t f = 3 * np;
        for (int l = 1; l <= L; ++l) {
            h.fo[l] = f;
            f += (int64_t)h.lv[l - 1].neven * S;
        }
        int64_t acc = 0;
        for (int k = 0; k < nstage; ++k) {
            h.begin[k] = acc;
            int nblk;
            if (k < 2 * L) nblk = (k & 1) ? h.lv[k >> 1].neven : h.lv[k >> 1].nodd;
            else if (k == 2 * L) nblk = 1;
            else if (k < 3 * L) nblk = h.lv[3 * L - k].nodd;
            else nblk = h.lv[0].nodd;   // E_0, C_0
            // the sparse stages B_0 and E_0 keep 32 rows
            const bool sparse = L > 0 && (k == 1 || k == 3 * L);
            const bool low = !sparse && nblk * ntile * ns <= P.low_tiles;
            h.tiles[k] = low ? (S + kLowRows - 1) / kLowRows : ntile;
            acc += (int64_t)nblk * h.tiles[k] * ns;
        }
        h.begin[nstage] = acc;
    }
    __syncthreads();
    const int64_t total = h.begin[nstage];
    auto live = [&](int64_t s) -> bool {
        return mask_has(a.live_mask, s) && !(a.skip && a.skip[s * a.skip_stride] != 0);
    };

    if (w == kTmaConsumerWarps) {
        // ------------------------------------------------------------------ producer
        if (lane == 0) {
            uint32_t slot = 0, ph = 0;
            int k = 0;
            uint64_t issued = 0;
            TileJob t;
            for (int64_t g = blockIdx.x; g < total; g += gridDim.x) {
                decode_tile(g, k, h, t);
                if (!live(t.s)) continue;
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    if (m >= t.nmat) break;
                    const int cols = t.low ? 4 * kCols : kCols;
                    for (int ch = 0; ch * cols < S; ++ch) {
                        if (!mbar_wait(&empty[slot], ph ^ 1)) atomicCAS(a.err, 0, KORE_DEVERR_FLAG);
                        mbar_arrive_expect_tx(&full[slot], CHUNK);
                        tma_load_4d(ring + (size_t)slot * CHUNK, &P.maps[t.map[m] + (t.low ? 4 : 0)], &full[slot],
                                    2 * t.r0, ch * cols, (int)t.mblk[m], (int)t.s);
                        ++issued;
                        if (++slot == (uint32_t)nst) { slot = 0; ph ^= 1; }
                    }
                }
            }
            // every copy has landed before the CTA may exit (normally already consumed)
            const uint64_t first = issued > (uint64_t)nst ? issued - nst : 0;
            for (uint64_t i = first; i < issued; ++i)
                if (!mbar_wait(&full[i % nst], (uint32_t)((i / nst) & 1))) atomicCAS(a.err, 0, KORE_DEVERR_FLAG);
        }
        return;
    }
    // ---------------------------------------------------------------------- consumers
    // Each warp follows the CTA's tiles on its own: it waits for and loads the entries of the
    // input vectors that its columns of the chunks multiply, consumes its columns of every
    // chunk of the ring, and leaves its partial sums in red; one named barrier per tile
    // gathers them, after which warp 0 reduces and writes the rows while the other warps go on.
    uint32_t slot = 0, ph = 0;
    int k = 0;
    TileJob t;
    int64_t i = 0;
    int64_t scaled = -1;     // the shift of bscale (an FP64 division, kept off the tiles' path)
    double bscale = 1.0;
    for (int64_t g = blockIdx.x; g < total; g += gridDim.x) {
        decode_tile(g, k, h, t);
        const int64_t s = t.s;
        C (*rd)[33] = red[i & 1];   // i counts the tiles worked on: two in a row never share
        if (live(s)) {
            ++i;
            C *vs = static_cast<C *>(a.vecs) + s * a.vec_stride;
            // level-0 couplings (B_0, E_0): this thread's padded entries are loaded before
            // the wait, as they do not depend on the sweep; lane = row, warp w = entries w + 8u
            const bool ell = (t.kind == 1 && t.l == 0) || t.kind == 4;
            const int64_t ebase = (t.blk * ntile + t.r0 / kTileRows) * (int64_t)a.ell_w * 32 + lane;
            const C *ellv = static_cast<const C *>(a.ell_val) + s * a.ell_stride;
            int ecol[kEllReg];
            C eval[kEllReg];
#pragma unroll
            for (int u = 0; u < kEllReg; ++u) {
                const int kk = w + u * kTmaConsumerWarps;
                const bool in = ell && kk < a.ell_w;
                ecol[u] = in ? __ldg(a.ell_col + ebase + (int64_t)kk * 32) : -1;
                eval[u] = in ? ldg(ellv + ebase + (int64_t)kk * 32) : czero<C>();
            }
            // rows this tile writes; the right-hand side does not depend on the sweep
            const int r = t.r0 + (t.low ? lane & 7 : lane);
            const int64_t p = t.blk * S + r;
            const bool wr = w == 0 && r < S && !(t.low && lane >= kLowRows);
            C zf = czero<C>();
            double2 prev = mk(0.0, 0.0);
            if ((t.from_b || ell) && scaled != s) {
                const double bn = a.bnorm[s];
                bscale = (bn > 0.0) ? 1.0 / bn : 1.0;
                scaled = s;
            }
            if (wr && ell) zf = from_c128<C>((a.rscale[s * np + p] * bscale) * a.b[s * np + p]);
            if (wr && (t.kind == 2 || t.kind == 3) && a.accumulate) prev = a.out[s * np + p];
            if (!ell && t.nmat > 0) {
                // this warp's slice of the input vectors.  A lane per vector waits for one of its
                // entries first, so that tiles far ahead poll little.
                if (!t.from_b && lane < t.nmat) wait_entry(vs + (lane ? t.in[1] : t.in[0]) + S - 1, a.err);
                __syncwarp();
                const int per = nvec / kTmaConsumerWarps;   // zeros past S: the chunks reach there
                const int ne = t.nmat * per;
                for (int e0 = 0; e0 < ne; e0 += 32 * kFill) {
                    C v[kFill];
                    int cv[kFill];   // column of the entry, + S for the second vector; -1: none
#pragma unroll
                    for (int u = 0; u < kFill; ++u) {
                        const int e = e0 + u * 32 + lane;
                        const int m = e >= per ? 1 : 0, rem = e - m * per;
                        const int c = (rem / kRun) * 4 * kRun + w * kRun + rem % kRun;
                        cv[u] = (e < ne) ? m * nvec + c : -1;
                        v[u] = czero<C>();
                        if (e < ne && c < S) {
                            if (t.from_b) {
                                const int64_t q = s * np + t.blk * S + c;
                                v[u] = from_c128<C>((a.rscale[q] * bscale) * a.b[q]);
                            } else v[u] = ld_entry(vs + (m ? t.in[1] : t.in[0]) + c);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < kFill; ++u)
                        if (cv[u] >= 0) {
                            if (!t.from_b && unset(v[u])) {
                                const int m = cv[u] >= nvec ? 1 : 0;
                                v[u] = wait_entry(vs + (m ? t.in[1] : t.in[0]) + cv[u] - m * nvec, a.err);
                            }
                            vbuf[cv[u]] = v[u];
                        }
                }
                __syncwarp();
            }
            if (wr && t.add >= 0) zf = ld_entry(vs + t.add + r);
            C sums[kAcc];
#pragma unroll
            for (int q = 0; q < kAcc; ++q) sums[q] = czero<C>();
            C &acc = sums[0];
            if (ell) {
                const C *z = vs + t.in[0];   // E_0 couples to x, B_0 to z
                C zv[kEllReg];
#pragma unroll
                for (int u = 0; u < kEllReg; ++u) zv[u] = ecol[u] >= 0 ? ld_entry(z + ecol[u]) : czero<C>();
#pragma unroll
                for (int u = 0; u < kEllReg; ++u)
                    if (ecol[u] >= 0) {
                        if (unset(zv[u])) zv[u] = wait_entry(z + ecol[u], a.err);
                        acc = cfma(acc, eval[u], zv[u]);
                    }
                for (int kk = w + kEllReg * kTmaConsumerWarps; kk < a.ell_w; kk += kTmaConsumerWarps) {
                    const int c = __ldg(a.ell_col + ebase + (int64_t)kk * 32);
                    if (c >= 0) acc = cfma(acc, ldg(ellv + ebase + (int64_t)kk * 32), wait_entry(z + c, a.err));
                }
            } else if (t.nmat > 0) {
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    if (m >= t.nmat) break;
                    // the warp's columns of a chunk; in low tiles of complex128 column
                    // 16 u + 4 w + lane / 8
                    const bool split = t.low && kSplit;
                    const C *vv = vbuf + m * nvec;
                    const int cols = t.low ? 4 * kCols : kCols;
                    for (int ch = 0; ch * cols < S; ++ch) {
                        if (!mbar_wait(&full[slot], ph)) atomicCAS(a.err, 0, KORE_DEVERR_FLAG);
                        const C *cb = reinterpret_cast<const C *>(ring + (size_t)slot * CHUNK);
                        const C *vc = vv + ch * cols;
                        if (split) {
                            const C *bc = cb + 4 * w * kLowRows + lane;
                            vc += 4 * w + (lane >> 3);
#pragma unroll
                            for (int u = 0; u < kCols / 4; ++u) acc = cfma(acc, bc[u * 16 * kLowRows], vc[16 * u]);
                        } else if (t.low) {
#pragma unroll
                            for (int h = 0; h < kCols / kRun; ++h) {
                                const int c0 = (4 * h + w) * kRun;
                                const C *bc = cb + c0 * kLowRows + (lane & 7);
#pragma unroll
                                for (int u = 0; u < kRun; ++u) acc = cfma(acc, bc[u * kLowRows], vc[c0 + u]);
                            }
                        } else if (kSplit) {
#pragma unroll
                            for (int h = 0; h < kCols / 16; ++h) {
                                const int c0 = 16 * h + 4 * w;
                                const C *bc = cb + c0 * kTileRows + lane;
#pragma unroll
                                for (int q = 0; q < kAcc; ++q) sums[q] = cfma(sums[q], bc[q * kTileRows], vc[c0 + q]);
                            }
                        } else if (!kHalf || (ch & 1) == (w >> 1)) {
                            const int c0 = kHalf ? (w & 1) * kRun : w * kRun;
                            const C *bc = cb + c0 * kTileRows + lane;
#pragma unroll
                            for (int u = 0; u < kRun; ++u) acc = cfma(acc, bc[u * kTileRows], vc[c0 + u]);
                        }
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&empty[slot]);
                        if (++slot == (uint32_t)nst) { slot = 0; ph ^= 1; }
                    }
                }
            }
            if (kSplit && !ell) {   // the four column classes of a row
                if (t.low) {
                    acc = acc + shfl_xor(acc, 8);
                    acc = acc + shfl_xor(acc, 16);
                } else acc = (acc + sums[kAcc > 1 ? 1 : 0]) + (sums[kAcc > 2 ? 2 : 0] + sums[kAcc > 3 ? 3 : 0]);
            }
            rd[w][lane] = acc;
            named_sync(1, kTmaConsumers);
            if (w == 0) {
                C val = czero<C>();
#pragma unroll
                for (int q = 0; q < kTmaConsumerWarps; ++q) val = val + rd[q][lane];
                if (wr) {
                    if (t.add >= 0 && unset(zf)) zf = wait_entry(vs + t.add + r, a.err);
                    if (ell || t.add >= 0) val = zf - val;
                    st_entry(vs + t.out + r, val);
                    if (t.kind == 2 || t.kind == 3) {   // an entry of the solution
                        const double bn = a.bnorm[s];
                        const double2 d = ((bn > 0.0) ? bn : 1.0) * to_c128(val);
                        a.out[s * np + p] = a.accumulate ? prev + d : d;
                    }
                }
            }
        }
    }
}

// |v| of a double as the bits of its absolute value: for non-negative IEEE doubles the
// integer order is the numeric order, so maxima run on the integer units, not on the
// FP64 pipe, and a NaN (above +inf as bits) is kept instead of dropped as fmax drops it
__device__ __forceinline__ unsigned long long abs_bits(double v) {
    return (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
}
__device__ __forceinline__ unsigned long long warp_max_bits(unsigned long long v) {
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}

// True in every thread of the last CTA of a grid row to get here (the CTAs' earlier writes
// are then visible to it); *tick is 0 before and after the launch.
__device__ __forceinline__ bool last_cta(unsigned *tick, unsigned ctas) {
    __shared__ bool last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(tick, 1u) == ctas - 1;
        if (last) {
            *tick = 0;
            __threadfence();
        }
    }
    __syncthreads();
    return last;
}

// Set all bits of the sweep's vectors of shift s (st_entry), this CTA's share of them.
__device__ __forceinline__ void reset_vecs(void *vecs, int64_t bytes, int64_t s) {
    uint4 *v = reinterpret_cast<uint4 *>(static_cast<unsigned char *>(vecs) + s * bytes);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < bytes / 16; i += (int64_t)gridDim.x * blockDim.x)
        v[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
}

// What a sweep of the right-hand sides b needs first, per shift (grid y): ||b||_inf (a NaN
// does not count), the sweep's vectors set, and with ir the refinement state of a new
// application (a shift outside live_mask has nothing to refine).  Bound by its launch: one
// kernel here for two maxima kernels, a state kernel and a memset, and the check in the
// residual product's last CTA, took a solve of 480 unknowns in FP64 from 123 to 102 us and
// four mixed targets of a 5.8k-unknown shell from 74.9 to 68.5 ms.
__global__ void __launch_bounds__(256) k_begin(int64_t np, const double2 *__restrict__ v, double *__restrict__ part,
                                               double *__restrict__ bnorm, unsigned *tick, void *vecs, int64_t vbytes,
                                               IrState *ir, unsigned live_mask) {
    const int s = blockIdx.y;
    reset_vecs(vecs, vbytes, s);
    v += s * np;
    part += (int64_t)s * gridDim.x;
    unsigned long long mx = 0;
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < np; p += (int64_t)gridDim.x * blockDim.x) {
        const unsigned long long x = abs_bits(v[p].x), y = abs_bits(v[p].y);
        if (x <= 0x7ff0000000000000ull) mx = max(mx, x);
        if (y <= 0x7ff0000000000000ull) mx = max(mx, y);
    }
    __shared__ unsigned long long sm[8];
    mx = warp_max_bits(mx);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) mx = max(mx, sm[w]);
        part[blockIdx.x] = __longlong_as_double((long long)mx);
    }
    if (!last_cta(tick + s, gridDim.x)) return;
    mx = 0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) mx = max(mx, abs_bits(__ldcg(part + i)));
    mx = warp_max_bits(mx);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = mx;
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int w = 1; w < 8; ++w) mx = max(mx, sm[w]);
    bnorm[s] = __longlong_as_double((long long)mx);
    if (!ir) return;
    const bool on = mask_has(live_mask, s);
    ir[s].done = on ? 0 : 1;
    if (on) {
        ir[s].prev = 1e300;
        ir[s].applies += 1;
    }
}

// Sparse products y = B x, A x - lam B x and the refinement residual b - (A x - lam B x).
// On this GPU the FP64 pipe, not HBM, bounds them (about two FP64 multiply-adds per
// SM per clock), so A is stored as a real matrix split into real and imaginary
// coefficients (two multiply-adds per value instead of four for a complex entry),
// each row's real and imaginary segments summed separately and combined at the end.
// Rows are short (a few dozen values): one thread per row with kRowUnroll gathers in
// flight.  Splitting a row over 2 or 4 lanes costs FP64 additions to combine the
// partial sums, which take FP64-pipe issue slots like the products do (measured on
// the 240k-unknown shell: 4 lanes 179 ms, 2 lanes 140 ms, 1 lane 129 ms per solve).
// The tau-method boundary rows are dense over a radial expansion (hundreds of
// entries); rows with more than kKoreLongRow values (A + B) are listed at plan
// creation and done by a whole warp each in extra CTAs at the end of the grid, so that
// they do not hold back the CTAs of the short rows.
constexpr int kRowLanes = 1;   // threads per short row
constexpr int kRowUnroll = 4;

struct SpmvArgs {
    int64_t np;
    int S, K;               // padded block size, blocks: row p's columns lie in blocks p/S - 1 .. p/S + 1
    int mode;               // 0: y = B x.  1: y = A x - lam B x.  2: y = b - (A x - lam B x)
    int has_b;
    const int *srow, *smid, *scol;  // A split into real and imaginary coefficients (kore_plan::d_s*)
    const double *sval;
    const int *brow, *bcol;
    const double *bval;
    const int *long_rows;   // rows done by a warp each
    int nlong;
    int short_blocks;       // CTAs of the 4-lane part (the long-row CTAs follow)
    double2 lam;            // shift when sig is null
    const double2 *sig;     // per-shift shifts (shift = blockIdx.y)
    const double2 *x, *rhs;
    double2 *y;
    double *part;           // mode 2: per-CTA maxima of |y| and |x|, part[s * 2 gridDim.x + 2 blockIdx.x (+1)]
    const int *skip;        // shift s is skipped when skip[s * skip_stride] != 0
    int skip_stride;
    unsigned live_mask;     // shift s (< 32) is computed only when bit s is set
};

// The entries of x one CTA of short rows reads, staged in shared memory: columns
// [w0, w1) (block-aligned: the blocks of the CTA's rows and one on either side).  An
// entry outside the window (none for a plan, whose band check keeps every column in the
// neighbouring blocks) is read from global memory.
struct XWin {
    const double2 *__restrict__ sh;
    int64_t w0, w1;
    __device__ __forceinline__ double2 get(const double2 *__restrict__ x, int c) const {
        return (c >= w0 && c < w1) ? sh[c - w0] : __ldg(x + c);
    }
};

// acc += sum over the values sub, sub + LANES, ... of [e0, e1) of val[e] x[col[e]]
// (kRowUnroll loads in flight per lane, two FP64 multiply-adds per value); x entries from
// the window when one is given
template <int LANES, bool WIN>
__device__ __forceinline__ void seg_dot(const int *__restrict__ col, const double *__restrict__ val, int e0, int e1,
                                        int sub, const double2 *__restrict__ x, const XWin &xw, double2 &acc) {
    for (int e = e0 + sub; e < e1; e += LANES * kRowUnroll) {
        int c[kRowUnroll];
        double v[kRowUnroll];
#pragma unroll
        for (int u = 0; u < kRowUnroll; ++u) {
            const int q = e + u * LANES;
            c[u] = q < e1 ? __ldg(col + q) : -1;
            v[u] = q < e1 ? __ldg(val + q) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < kRowUnroll; ++u)
            if (c[u] >= 0) {
                const double2 xv = WIN ? xw.get(x, c[u]) : __ldg(x + c[u]);
                acc.x = fma(v[u], xv.x, acc.x);
                acc.y = fma(v[u], xv.y, acc.y);
            }
    }
}

// Partial sums of row p: the real-coefficient values of A (sr), its imaginary-coefficient
// values (si: A x = sr + i si) and B (sb).
template <int LANES, bool WIN>
__device__ __forceinline__ void row_dot(const SpmvArgs &a, int64_t p, int sub, const double2 *__restrict__ x,
                                        const XWin &xw, double2 &sr, double2 &si, double2 &sb) {
    if (a.mode != 0) {
        const int em = a.smid[p];
        seg_dot<LANES, WIN>(a.scol, a.sval, a.srow[p], em, sub, x, xw, sr);
        seg_dot<LANES, WIN>(a.scol, a.sval, em, a.srow[p + 1], sub, x, xw, si);
    }
    if (a.has_b) seg_dot<LANES, WIN>(a.bcol, a.bval, a.brow[p], a.brow[p + 1], sub, x, xw, sb);
}

// x entries of the window of a CTA of 256 short rows: at most (255 / S + 4) blocks
__host__ __device__ __forceinline__ int64_t spmv_window(int S) { return (int64_t)(255 / S + 4) * S; }

// Per-shift refinement tolerances of one application (shifts past 31 use the scalar).
struct ShiftTols {
    double t[32];
    int valid;
};

// The refinement's test, run by the last CTA of a shift's residual product: eta = ||r||_inf /
// (||M||_inf ||x||_inf + ||b||_inf) from the CTAs' maxima; stop when eta <= tol or when it no
// longer decreases (FP64 floor).
struct IrCheck {
    IrState *ir;             // null: no test
    const double *bnorm, *minf;
    double *rn;              // ||r||_inf for the next correction
    double tol;
    ShiftTols tols;
    unsigned *tick;
    void *vecs;              // the next sweep's vectors, set here
    int64_t vbytes;
};

__device__ __forceinline__ void ir_check(const IrCheck &c, int s, const double *part, int n) {
    // maxima of non-negative doubles as bits (a NaN among them stays, and is caught below)
    unsigned long long rb = 0, xb = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        rb = max(rb, abs_bits(__ldcg(part + 2 * i)));
        xb = max(xb, abs_bits(__ldcg(part + 2 * i + 1)));
    }
    rb = warp_max_bits(rb);
    xb = warp_max_bits(xb);
    __shared__ unsigned long long s0[8], s1[8];
    if ((threadIdx.x & 31) == 0) { s0[threadIdx.x >> 5] = rb; s1[threadIdx.x >> 5] = xb; }
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int w = 1; w < 8; ++w) { rb = max(rb, s0[w]); xb = max(xb, s1[w]); }
    const double rm = __longlong_as_double((long long)rb), xm = __longlong_as_double((long long)xb);
    const double den = c.minf[s] * xm + c.bnorm[s];
    const double tol = (c.tols.valid && s < 32) ? c.tols.t[s] : c.tol;
    // a NaN in r, x or b makes eta NaN (a NaN denominator must not read as converged)
    const double eta = (den == 0.0) ? 0.0 : rm / den;
    IrState *st = c.ir + s;
    if (!(eta == eta)) {
        st->nan = 1;
        st->done = 1;
        return;
    }
    if (eta <= tol || eta > 0.9 * st->prev) {
        st->done = 1;
        st->eta_max = fmax(st->eta_max, eta);
        return;
    }
    st->prev = eta;
    st->iters += 1;
    st->iters_cur += 1;
    c.rn[s] = rm;
}

__global__ void __launch_bounds__(256) k_spmv(const SpmvArgs a, const __grid_constant__ IrCheck chk) {
    extern __shared__ double2 xsh[];   // spmv_window(S) entries
    const int64_t s = blockIdx.y;
    if (!mask_has(a.live_mask, s) || (a.skip && a.skip[s * a.skip_stride])) return;
    const int64_t np = a.np;
    const double2 *x = a.x + s * np;
    double2 *y = a.y + s * np;
    const double2 *rhs = a.rhs ? a.rhs + s * np : nullptr;
    const double2 lam = a.sig ? a.sig[s] : a.lam;
    unsigned long long rmax = 0, xmax = 0;
    auto finish = [&](int64_t p, double2 sr, double2 si, double2 sb) {
        const double2 sa = mk(sr.x - si.y, sr.y + si.x);   // A x = sr + i si
        double2 v = (a.mode == 0) ? sb : sa - lam * sb;
        if (a.mode == 2) {
            v = rhs[p] - v;
            const double2 xp = x[p];
            rmax = max(rmax, max(abs_bits(v.x), abs_bits(v.y)));
            xmax = max(xmax, max(abs_bits(xp.x), abs_bits(xp.y)));
        }
        y[p] = v;
    };
    if ((int)blockIdx.x < a.short_blocks) {
        static_assert(kRowLanes == 1, "one thread per short row");
        // stage the x entries of the blocks this CTA's rows couple to (coalesced), so the
        // rows' gathers hit shared memory instead of waiting on L2
        const int64_t r0 = blockIdx.x * (int64_t)blockDim.x;
        const int64_t rl = ((r0 + blockDim.x < np) ? r0 + blockDim.x : np) - 1;
        const int64_t b0 = (r0 / a.S > 0) ? r0 / a.S - 1 : 0;
        const int64_t b1 = (rl / a.S + 1 < a.K) ? rl / a.S + 1 : a.K - 1;
        XWin xw{xsh, b0 * a.S, (b1 + 1) * a.S};
        for (int64_t c = xw.w0 + threadIdx.x; c < xw.w1; c += blockDim.x) xsh[c - xw.w0] = __ldg(x + c);
        __syncthreads();
        const int64_t p = r0 + threadIdx.x;
        bool live = p < np;
        if (live) {
            const int len = (a.srow[p + 1] - a.srow[p]) + (a.has_b ? a.brow[p + 1] - a.brow[p] : 0);
            live = len <= kKoreLongRow;
        }
        if (live) {
            double2 sr = mk(0.0, 0.0), si = mk(0.0, 0.0), sb = mk(0.0, 0.0);
            row_dot<1, true>(a, p, 0, x, xw, sr, si, sb);
            finish(p, sr, si, sb);
        }
    } else {
        const int lane = threadIdx.x & 31;
        const int wid = (blockIdx.x - a.short_blocks) * (blockDim.x >> 5) + (threadIdx.x >> 5);
        if (wid < a.nlong) {
            const int64_t p = a.long_rows[wid];
            double2 sr = mk(0.0, 0.0), si = mk(0.0, 0.0), sb = mk(0.0, 0.0);
            row_dot<32, false>(a, p, lane, x, XWin{nullptr, 0, 0}, sr, si, sb);
            sr = warp_sum(sr);
            si = warp_sum(si);
            sb = warp_sum(sb);
            if (lane == 0) finish(p, sr, si, sb);
        }
    }
    if (a.mode == 2) {
        rmax = warp_max_bits(rmax);
        xmax = warp_max_bits(xmax);
        __shared__ unsigned long long sm[2][8];
        if ((threadIdx.x & 31) == 0) { sm[0][threadIdx.x >> 5] = rmax; sm[1][threadIdx.x >> 5] = xmax; }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < (int)(blockDim.x >> 5); ++w) { rmax = max(rmax, sm[0][w]); xmax = max(xmax, sm[1][w]); }
            a.part[s * 2 * gridDim.x + 2 * blockIdx.x] = __longlong_as_double((long long)rmax);
            a.part[s * 2 * gridDim.x + 2 * blockIdx.x + 1] = __longlong_as_double((long long)xmax);
        }
        if (chk.ir) {
            reset_vecs(chk.vecs, chk.vbytes, s);
            if (last_cta(chk.tick + s, gridDim.x)) ir_check(chk, (int)s, a.part + s * 2 * gridDim.x, (int)gridDim.x);
        }
    }
}

// padded[s * np + p] = orig[s * n + slot2orig[p]] (0 on pad slots); shift = blockIdx.y
__global__ void k_gather(int64_t np, int64_t n, const int64_t *__restrict__ s2o, const double2 *__restrict__ orig,
                         double2 *__restrict__ padded) {
    const int64_t s = blockIdx.y;
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < np; p += (int64_t)gridDim.x * blockDim.x) {
        const int64_t o = s2o[p];
        padded[s * np + p] = (o >= 0) ? orig[s * n + o] : mk(0.0, 0.0);
    }
}
__global__ void k_scatter(int64_t np, int64_t n, const int64_t *__restrict__ s2o, const double2 *__restrict__ padded,
                          double2 *__restrict__ orig) {
    const int64_t s = blockIdx.y;
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < np; p += (int64_t)gridDim.x * blockDim.x) {
        const int64_t o = s2o[p];
        if (o >= 0) orig[s * n + o] = padded[s * np + p];
    }
}

template <typename C>
size_t tma_smem(int S, int nst, int chunk) {
    const int kCols = chunk / (kTileRows * (int)sizeof(C));
    const int nvec = (S + 4 * kCols - 1) / (4 * kCols) * (4 * kCols);
    return (size_t)nst * chunk + 2 * (size_t)nst * sizeof(uint64_t) + 2 * (size_t)nvec * sizeof(C);
}

template <typename C>
void (*sweep_kernel(TmaVariant v))(const SweepTmaParams) {
    if (v.chunk == 8192)
        return v.cps == 2 ? k_sweep_tma<C, 2, 8192> : v.cps == 4 ? k_sweep_tma<C, 4, 8192> : k_sweep_tma<C, 3, 8192>;
    return v.cps == 2 ? k_sweep_tma<C, 2, 16384> : v.cps == 4 ? k_sweep_tma<C, 4, 16384> : k_sweep_tma<C, 3, 16384>;
}

// Sweep arguments of the plan's factors for `nshift` shifts starting at shift 0; the
// caller sets the vectors, counters and flags.
SweepArgs sweep_args(const kore_plan *p, int nshift) {
    SweepArgs a;
    a.K = p->K; a.S = p->S; a.nlev = p->nlev; a.nshift = nshift; a.levs = p->d_lev;
    a.Dinv = p->d_Dinv; a.G = p->d_Gm; a.H = p->d_Hm; a.LU = p->d_LU;
    a.f_stride = p->f_stride(); a.lu_stride = p->lu_stride();
    a.ell_col = p->d_ell_col; a.ell_val = p->d_ell_val; a.ell_w = p->ell_w; a.ell_stride = p->ell_stride();
    a.rscale = p->d_rscale;
    a.vec_stride = p->sweep_vec_elems();
    a.live_mask = ~0u;
    return a;
}

// Largest number of 32-row tiles of a stage that takes 8-row tiles (kLowRows).  A lone tile
// of complex128 fills its SM's FP64 pipe, so splitting pays while there are fewer tiles than
// SMs; complex64 tiles wait on their chunks and still gain with two per SM.  Whole solves
// with limits 0, 40, 76, 101, 152 and 304: 72k shell in complex128 918, 771, 756, 742, 721,
// 730 us; 240k shell in complex64 (7 sweeps) 5.26, 5.06, 4.98, 4.98, 4.90, 4.88 ms.
int sweep_low_tiles(const kore_plan *p) { return p->prec == KORE_PREC_FP64 ? p->num_sms : 2 * p->num_sms; }

// What a launch of a variant needs besides its arguments.  The plan keeps its last one: maps
// and occupancy depend on the variant, the factors' storage and the number of shifts alone,
// and encoding and asking for them takes the host longer than a small sweep runs.
struct SweepLaunch {
    int prec, nshift, cps, chunk, occ;
    size_t smem;
    SweepTmaParams P;
};

template <typename C>
int prepare_sweep(const kore_plan *p, TmaVariant v, int ns, SweepLaunch &l) {
    const int rb = (int)sizeof(C) / 2;
    if (v.chunk != 8192 && v.chunk != 16384) return KORE_EINVAL;
    const int kCols = v.chunk / (kTileRows * (int)sizeof(C));
    SweepTmaParams &P = l.P;
    for (int low = 0; low < 2; ++low) {
        const int rows = low ? kLowRows : kTileRows, cols = low ? 4 * kCols : kCols, o = 4 * low;
        KORE_TRY(kore_encode_block_map(&P.maps[o + kMapDinv], p->d_Dinv, rb, p->S, p->K, ns, p->f_stride(), rows, cols));
        KORE_TRY(kore_encode_block_map(&P.maps[o + kMapG], p->d_Gm, rb, p->S, p->K, ns, p->f_stride(), rows, cols));
        KORE_TRY(kore_encode_block_map(&P.maps[o + kMapH], p->d_Hm, rb, p->S, p->K, ns, p->f_stride(), rows, cols));
        KORE_TRY(kore_encode_block_map(&P.maps[o + kMapLU], p->d_LU, rb, p->S, p->lu_mats, ns, p->lu_stride(), rows,
                                       cols));
    }
    P.low_tiles = sweep_low_tiles(p);
    // ring depth: as many slots as fit cps CTAs in the SM's shared memory
    int smem_sm = 0, smem_blk = 0;
    KORE_CUDA_TRY(cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, p->device));
    KORE_CUDA_TRY(cudaDeviceGetAttribute(&smem_blk, cudaDevAttrMaxSharedMemoryPerBlockOptin, p->device));
    void (*kern)(const SweepTmaParams) = sweep_kernel<C>(v);
    cudaFuncAttributes fa;
    KORE_CUDA_TRY(cudaFuncGetAttributes(&fa, kern));
    const size_t static_smem = fa.sharedSizeBytes + 1024;   // + the per-CTA reserve of the SM
    const size_t budget = std::min<size_t>((size_t)smem_sm / v.cps - static_smem,
                                           (size_t)smem_blk - fa.sharedSizeBytes);
    int nst = kMaxRing;
    while (nst > 2 && tma_smem<C>(p->S, nst, v.chunk) > budget) --nst;
    if (tma_smem<C>(p->S, nst, v.chunk) > budget) return KORE_EINVAL;
    P.nst = nst;
    l.smem = tma_smem<C>(p->S, nst, v.chunk);
    KORE_TRY(kore_allow_max_dyn_smem(kern, p->device));
    int occ = 0;
    KORE_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kTmaThreads, l.smem));
    if (occ < 1) return KORE_EINVAL;
    l.occ = std::min(occ, v.cps);
    l.prec = p->prec; l.nshift = ns; l.cps = v.cps; l.chunk = v.chunk;
    return KORE_OK;
}

// The cooperative launch of a prepared k_sweep_tma on the vectors that the kernel before it set
template <typename C>
int launch_prepared(SweepLaunch &l, const SweepArgs &a, int num_sms, cudaStream_t st) {
    l.P.a = a;
    void *args[] = {&l.P};
    KORE_CUDA_TRY(cudaLaunchCooperativeKernel((const void *)sweep_kernel<C>(TmaVariant{l.cps, l.chunk}),
                                              dim3(num_sms * l.occ), dim3(kTmaThreads), args, l.smem, st));
    KORE_LAUNCHED(1);
    return KORE_OK;
}

// The same on the plan's own stream, prepared when the plan's last one was of another shape
template <typename C>
int launch_sweep(kore_plan *p, const SweepArgs &a, TmaVariant v) {
    SweepLaunch *l = static_cast<SweepLaunch *>(p->sweep_launch.get());
    if (!l || l->prec != p->prec || l->nshift != a.nshift || l->cps != v.cps || l->chunk != v.chunk) {
        std::shared_ptr<SweepLaunch> made = std::make_shared<SweepLaunch>();
        KORE_TRY(prepare_sweep<C>(p, v, a.nshift, *made));
        p->sweep_launch = made;
        l = made.get();
    }
    return launch_prepared<C>(*l, a, p->num_sms, p->stream);
}

// bytes of one shift's sweep vectors (16-byte entries or pairs: S is a multiple of 4)
int64_t vec_bytes(const kore_plan *p) {
    return p->sweep_vec_elems() * (int64_t)(p->prec == KORE_PREC_FP64 ? sizeof(double2) : sizeof(float2));
}

// Autotuner of the sweep's variant (CTAs per SM, chunk size), keyed on the plan's shape: the first
// non-accumulating sweep of a shape (padded block size, blocks, width of the level-0
// coupling rows, precision, shifts) times every variant on its own work (a
// non-accumulating sweep gives the same result each time it runs) and keeps the fastest
// for every later sweep of that shape in the process.
struct TuneKey {
    int S, K, ell_w, prec, nshift;
    bool operator<(const TuneKey &o) const {
        return std::tie(S, K, ell_w, prec, nshift) < std::tie(o.S, o.K, o.ell_w, o.prec, o.nshift);
    }
};
std::mutex g_tune_mu;
std::map<TuneKey, TmaVariant> g_tune;
TmaVariant g_force{0, 0};   // kore_sweep_variant: every sweep uses it instead of the autotuner's choice

template <typename C>
int reset_and_sweep(kore_plan *p, const SweepArgs &a, TmaVariant v) {
    KORE_CUDA_TRY(cudaMemsetAsync(a.vecs, 0xff, (size_t)a.nshift * vec_bytes(p), p->stream));
    return launch_sweep<C>(p, a, v);
}

template <typename C>
int tune_sweep(kore_plan *p, const SweepArgs &a, TmaVariant *best) {
    cudaEvent_t e0, e1;
    KORE_CUDA_TRY(cudaEventCreate(&e0));
    KORE_CUDA_TRY(cudaEventCreate(&e1));
    float best_ms = 1e30f;
    int rc = KORE_OK;
    *best = kTmaDefault;
    for (const TmaVariant v : kTmaVariants) {
        float ms = 0.f;
        for (int rep = 0; rep < 2 && rc == KORE_OK; ++rep) {   // the second run is timed
            if (cudaEventRecord(e0, p->stream) != cudaSuccess) rc = KORE_ECUDA;
            if (rc == KORE_OK) rc = reset_and_sweep<C>(p, a, v);
            if (rc == KORE_OK && cudaEventRecord(e1, p->stream) != cudaSuccess) rc = KORE_ECUDA;
            if (rc == KORE_OK && cudaEventSynchronize(e1) != cudaSuccess) rc = KORE_ECUDA;
            if (rc == KORE_OK && cudaEventElapsedTime(&ms, e0, e1) != cudaSuccess) rc = KORE_ECUDA;
        }
        if (rc == KORE_EINVAL) { rc = KORE_OK; continue; }   // the variant does not fit this shape
        if (rc != KORE_OK) break;
        if (ms < best_ms) { best_ms = ms; *best = v; }
    }
    // the chosen variant runs last, so the sweep's outputs are its own
    if (rc == KORE_OK) rc = reset_and_sweep<C>(p, a, *best);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return rc;
}

int sweep(kore_plan *p, const double2 *b, const double *bnorm, double2 *x, int accumulate, const int *skip,
          unsigned live_mask) {
    if (p->prof) KORE_TRY(kore_prof_mark(p, 0, true));
    SweepArgs a = sweep_args(p, p->nshift);
    a.live_mask = live_mask;
    a.b = b; a.bnorm = bnorm;
    a.vecs = p->d_sweep;
    a.out = x; a.accumulate = accumulate; a.err = p->d_err;
    a.skip = skip; a.skip_stride = (int)(sizeof(IrState) / sizeof(int));
    a.count = &p->d_ir->sweeps; a.count_total = &p->d_ir->sweeps_total;
    const bool fp64 = p->prec == KORE_PREC_FP64;
    const TuneKey key{p->S, p->K, p->ell_w, p->prec, p->nshift};
    TmaVariant v{0, 0};
    bool forced = false;
    {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        auto it = g_tune.find(key);
        if (g_force.cps != 0) { v = g_force; forced = true; }
        else if (it != g_tune.end()) v = it->second;
    }
    int s;
    if (v.cps == 0 && !accumulate && !forced) {
        s = fp64 ? tune_sweep<double2>(p, a, &v) : tune_sweep<float2>(p, a, &v);
        if (s == KORE_OK) {
            std::lock_guard<std::mutex> lk(g_tune_mu);
            g_tune[key] = v;
        }
    } else {
        if (v.cps == 0) v = kTmaDefault;
        s = fp64 ? launch_sweep<double2>(p, a, v) : launch_sweep<float2>(p, a, v);
    }
    p->sweep_cps = v.cps;
    p->sweep_chunk = v.chunk;
    if (p->prof) KORE_TRY(kore_prof_mark(p, 0, false));
    return s;
}

}  // namespace

extern "C" int kore_sweep_variant(int ctas_per_sm, int chunk_bytes) {
    bool ok = ctas_per_sm == 0 && chunk_bytes == 0;
    for (const TmaVariant v : kTmaVariants) ok = ok || (v.cps == ctas_per_sm && v.chunk == chunk_bytes);
    if (!ok) return KORE_EINVAL;
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_force = TmaVariant{ctas_per_sm, chunk_bytes};
    return KORE_OK;
}

namespace {

unsigned begin_grid(const kore_plan *p) { return std::min<unsigned>(kore_div_up(p->np, 256), 2u * p->num_sms); }

// CTAs of one sparse product: the 4-lane part, then 8 long rows per CTA
unsigned spmv_short_blocks(int64_t np) { return kore_div_up(np * kRowLanes, 256); }
unsigned spmv_grid(const kore_plan *p) { return spmv_short_blocks(p->np) + kore_div_up(p->nlong, 8); }
size_t spmv_smem(const kore_plan *p) { return (size_t)spmv_window(p->S) * sizeof(double2); }

SpmvArgs spmv_args(const kore_plan *p, int mode, const double2 *x, double2 *y) {
    SpmvArgs a;
    a.np = p->np; a.S = p->S; a.K = p->K; a.mode = mode; a.has_b = p->has_b ? 1 : 0;
    a.srow = p->d_srow; a.smid = p->d_smid; a.scol = p->d_scol; a.sval = p->d_sval;
    a.brow = p->d_brow; a.bcol = p->d_bcol; a.bval = p->d_bval;
    a.long_rows = p->d_long_rows; a.nlong = p->nlong; a.short_blocks = (int)spmv_short_blocks(p->np);
    a.lam = mk(0.0, 0.0); a.sig = nullptr;
    a.x = x; a.rhs = nullptr; a.y = y; a.part = nullptr;
    a.skip = nullptr; a.skip_stride = 0;
    a.live_mask = ~0u;
    return a;
}

}  // namespace

int kore_spmv_prepare(kore_plan *p) {
    // the x window of a CTA exceeds the default 48 KB of shared memory for S > 760
    return kore_allow_max_dyn_smem(k_spmv, p->device);
}

int kore_spmv_b(kore_plan *p, const double2 *x, double2 *y) {
    if (!p->has_b) return KORE_EINVAL;
    if (p->prof) KORE_TRY(kore_prof_mark(p, 2, true));
    k_spmv<<<spmv_grid(p), 256, spmv_smem(p), p->stream>>>(spmv_args(p, 0, x, y), IrCheck{});
    KORE_LAUNCHED(1);
    if (p->prof) KORE_TRY(kore_prof_mark(p, 2, false));
    KORE_CUDA_TRY(cudaGetLastError());
    return KORE_OK;
}

int kore_spmv_b_shifts(kore_plan *p, const double2 *x, double2 *y, unsigned live_mask) {
    if (!p->has_b) return KORE_EINVAL;
    if (p->prof) KORE_TRY(kore_prof_mark(p, 2, true));
    SpmvArgs a = spmv_args(p, 0, x, y);
    a.live_mask = live_mask;
    k_spmv<<<dim3(spmv_grid(p), std::max(1, p->nshift)), 256, spmv_smem(p), p->stream>>>(a, IrCheck{});
    KORE_LAUNCHED(1);
    if (p->prof) KORE_TRY(kore_prof_mark(p, 2, false));
    KORE_CUDA_TRY(cudaGetLastError());
    return KORE_OK;
}

int kore_spmv_a_shifts(kore_plan *p, const double2 *x, double2 *y, unsigned live_mask) {
    if (p->prof) KORE_TRY(kore_prof_mark(p, 2, true));
    SpmvArgs a = spmv_args(p, 1, x, y);   // A x - 0 B x
    a.has_b = 0;
    a.live_mask = live_mask;
    k_spmv<<<dim3(spmv_grid(p), std::max(1, p->nshift)), 256, spmv_smem(p), p->stream>>>(a, IrCheck{});
    KORE_LAUNCHED(1);
    if (p->prof) KORE_TRY(kore_prof_mark(p, 2, false));
    KORE_CUDA_TRY(cudaGetLastError());
    return KORE_OK;
}

int kore_spmv_pencil(kore_plan *p, double lre, double lim, const double2 *x, double2 *y) {
    SpmvArgs a = spmv_args(p, 1, x, y);
    a.lam = mk(lre, lim);
    k_spmv<<<spmv_grid(p), 256, spmv_smem(p), p->stream>>>(a, IrCheck{});
    KORE_LAUNCHED(1);
    KORE_CUDA_TRY(cudaGetLastError());
    return KORE_OK;
}

int kore_gather(kore_plan *p, const double2 *orig, double2 *padded) {
    const unsigned grid = std::min<unsigned>(kore_div_up(p->np, 256), 2048u);
    k_gather<<<grid, 256, 0, p->stream>>>(p->np, p->n, p->d_slot2orig, orig, padded);
    KORE_LAUNCHED(1);
    KORE_CUDA_TRY(cudaGetLastError());
    return KORE_OK;
}

int kore_scatter(kore_plan *p, const double2 *padded, double2 *orig) {
    const unsigned grid = std::min<unsigned>(kore_div_up(p->np, 256), 2048u);
    k_scatter<<<grid, 256, 0, p->stream>>>(p->np, p->n, p->d_slot2orig, padded, orig);
    KORE_LAUNCHED(1);
    KORE_CUDA_TRY(cudaGetLastError());
    return KORE_OK;
}

int kore_gather_shifts(kore_plan *p, const double2 *orig, double2 *padded) {
    const unsigned grid = std::min<unsigned>(kore_div_up(p->np, 256), 2048u);
    k_gather<<<dim3(grid, p->nshift), 256, 0, p->stream>>>(p->np, p->n, p->d_slot2orig, orig, padded);
    KORE_LAUNCHED(1);
    KORE_CUDA_TRY(cudaGetLastError());
    return KORE_OK;
}

int kore_scatter_shifts(kore_plan *p, const double2 *padded, double2 *orig) {
    const unsigned grid = std::min<unsigned>(kore_div_up(p->np, 256), 2048u);
    k_scatter<<<dim3(grid, p->nshift), 256, 0, p->stream>>>(p->np, p->n, p->d_slot2orig, padded, orig);
    KORE_LAUNCHED(1);
    KORE_CUDA_TRY(cudaGetLastError());
    return KORE_OK;
}

namespace {

// Vectors stored side by side: entry o of shift s's vector at orig[ld o + s] (shared: one
// vector for all).  CTA = 32 padded rows x 8 shifts at a time through shared memory, so that
// both sides are read and written in runs.
__global__ void __launch_bounds__(256) k_gather_cols(int64_t np, int ns, const int64_t *__restrict__ s2o,
                                                     const double2 *__restrict__ orig, int ld, int shared,
                                                     double2 *__restrict__ padded) {
    __shared__ double2 t[8][33];
    const int64_t p0 = blockIdx.x * 32LL;
    for (int s0 = 0; s0 < ns; s0 += 8) {
        {
            const int s = s0 + (threadIdx.x & 7), r = threadIdx.x >> 3;
            const int64_t o = p0 + r < np ? s2o[p0 + r] : -1;
            t[threadIdx.x & 7][r] = (o >= 0 && s < ns) ? orig[o * ld + (shared ? 0 : s)] : mk(0.0, 0.0);
        }
        __syncthreads();
        const int s = s0 + (threadIdx.x >> 5), r = threadIdx.x & 31;
        if (s < ns && p0 + r < np) padded[s * np + p0 + r] = t[threadIdx.x >> 5][r];
        __syncthreads();
    }
}
__global__ void __launch_bounds__(256) k_scatter_cols(int64_t np, int ns, const int64_t *__restrict__ s2o,
                                                      const double2 *__restrict__ padded, double2 *__restrict__ orig,
                                                      int ld) {
    __shared__ double2 t[8][33];
    const int64_t p0 = blockIdx.x * 32LL;
    for (int s0 = 0; s0 < ns; s0 += 8) {
        {
            const int s = s0 + (threadIdx.x >> 5), r = threadIdx.x & 31;
            if (s < ns && p0 + r < np) t[threadIdx.x >> 5][r] = padded[s * np + p0 + r];
        }
        __syncthreads();
        const int s = s0 + (threadIdx.x & 7), r = threadIdx.x >> 3;
        const int64_t o = p0 + r < np ? s2o[p0 + r] : -1;
        if (o >= 0 && s < ns) orig[o * ld + s] = t[threadIdx.x & 7][r];
        __syncthreads();
    }
}
__global__ void k_check_finite(const double2 *__restrict__ v, int64_t n, int *flag) {
    bool bad = false;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double2 x = v[i];
        bad = bad || (__double2hiint(x.x) & 0x7ff00000) == 0x7ff00000 || (__double2hiint(x.y) & 0x7ff00000) == 0x7ff00000;
    }
    if (bad) *flag = 1;
}

}  // namespace

int kore_gather_cols(kore_plan *p, const double2 *orig, int ld, bool shared, double2 *padded) {
    k_gather_cols<<<kore_div_up(p->np, 32), 256, 0, p->stream>>>(p->np, p->nshift, p->d_slot2orig, orig, ld, shared, padded);
    KORE_LAUNCHED(1);
    KORE_CUDA_TRY(cudaGetLastError());
    return KORE_OK;
}
int kore_scatter_cols(kore_plan *p, const double2 *padded, double2 *orig, int ld) {
    k_scatter_cols<<<kore_div_up(p->np, 32), 256, 0, p->stream>>>(p->np, p->nshift, p->d_slot2orig, padded, orig, ld);
    KORE_LAUNCHED(1);
    KORE_CUDA_TRY(cudaGetLastError());
    return KORE_OK;
}
int kore_check_finite(kore_plan *p, const double2 *v, int64_t n, int *flag) {
    KORE_CUDA_TRY(cudaMemsetAsync(flag, 0, sizeof(int), p->stream));
    k_check_finite<<<std::min<unsigned>(kore_div_up(n, 256), 1024u), 256, 0, p->stream>>>(v, n, flag);
    KORE_LAUNCHED(1);
    KORE_CUDA_TRY(cudaGetLastError());
    return KORE_OK;
}

namespace {

__global__ void k_ir_end(IrState *st, int nshift) {
    const int s = threadIdx.x;
    if (s >= nshift) return;
    if (st[s].iters_cur > st[s].iters_max) st[s].iters_max = st[s].iters_cur;
    // the loop ran out of corrections before the test passed: report the last measured
    // eta (taken before the final correction, so an upper estimate)
    if (!st[s].done && st[s].iters_cur > 0) st[s].eta_max = fmax(st[s].eta_max, st[s].prev);
    st[s].iters_cur = 0;
}

}  // namespace

// Mixed precision: the refinement loop runs without host synchronisation.  Its length
// is bounded (kIrMax corrections); each step is a residual kernel, whose last CTA of a shift
// runs the convergence check, and a correction sweep, and once the check marks a shift done
// the remaining work of that shift is skipped (kernels return at once when every
// shift is done).
constexpr int kIrMax = 6;
int kore_apply_inverse(kore_plan *p, const double2 *b, double2 *x, double tol, unsigned live_mask,
                       const double *shift_tols) {
    if (!p->factored) return KORE_ENOTFACTORED;
    double *bn = p->d_bn, *rn = p->d_rn;
    const int ns = p->nshift;
    const bool mixed = p->prec == KORE_PREC_MIXED;
    k_begin<<<dim3(begin_grid(p), ns), 256, 0, p->stream>>>(p->np, b, p->d_part, bn, p->d_tick, p->d_sweep, vec_bytes(p),
                                                            mixed ? p->d_ir : nullptr, live_mask);
    KORE_LAUNCHED(1);
    KORE_TRY(sweep(p, b, bn, x, 0, nullptr, live_mask));
    if (!mixed) return KORE_OK;
    if (!(tol > 0.0)) tol = 1e-14;
    IrCheck chk{};
    chk.ir = p->d_ir; chk.bnorm = bn; chk.minf = p->d_minf; chk.rn = rn; chk.tol = tol;
    chk.tick = p->d_tick; chk.vecs = p->d_sweep; chk.vbytes = vec_bytes(p);
    chk.tols.valid = shift_tols ? 1 : 0;
    for (int s = 0; s < 32 && shift_tols && s < p->nshift; ++s)
        chk.tols.t[s] = (shift_tols[s] > 0.0) ? shift_tols[s] : tol;
    const int skip_stride = (int)(sizeof(IrState) / sizeof(int));
    const unsigned grid = spmv_grid(p);
    SpmvArgs ra = spmv_args(p, 2, x, p->d_rb);
    ra.sig = p->d_sigma; ra.rhs = b; ra.part = p->d_part; ra.skip = &p->d_ir->done; ra.skip_stride = skip_stride;
    ra.live_mask = live_mask;
    for (int it = 0; it < kIrMax; ++it) {
        if (p->prof) KORE_TRY(kore_prof_mark(p, 2, true));
        k_spmv<<<dim3(grid, ns), 256, spmv_smem(p), p->stream>>>(ra, chk);
        KORE_LAUNCHED(1);
        if (p->prof) KORE_TRY(kore_prof_mark(p, 2, false));
        KORE_TRY(sweep(p, p->d_rb, rn, x, 1, &p->d_ir->done, live_mask));
    }
    k_ir_end<<<1, ns, 0, p->stream>>>(p->d_ir, ns);
    KORE_LAUNCHED(1);
    KORE_CUDA_TRY(cudaGetLastError());
    return KORE_OK;
}

int kore_ir_reset(kore_plan *p) {
    // everything but the lifetime sweep counters
    KORE_CUDA_TRY(cudaMemset2DAsync(p->d_ir, sizeof(IrState), 0, offsetof(IrState, sweeps_total), std::max(1, p->nshift),
                                    p->stream));
    return KORE_OK;
}

// Aggregate over the factorised shifts: sweep counts of shift 0 (every launch counts
// there), worst refinement count and eta, NaN in any shift.
int kore_ir_read(kore_plan *p, IrState *out, int *err) {
    // through the plan's pinned buffer, with the error flag: one wait
    const int ns = std::max(1, p->nshift);
    std::vector<IrState> all(ns);
    const size_t bytes = ns * sizeof(IrState);
    IrState *h = 8 + bytes <= 8192 * sizeof(double) ? reinterpret_cast<IrState *>(p->h_red + 1) : all.data();
    KORE_CUDA_TRY(cudaMemcpyAsync(h, p->d_ir, bytes, cudaMemcpyDeviceToHost, p->stream));
    if (err) KORE_CUDA_TRY(cudaMemcpyAsync(p->h_red, p->d_err, sizeof(int), cudaMemcpyDeviceToHost, p->stream));
    KORE_CUDA_TRY(cudaStreamSynchronize(p->stream));
    if (h != all.data()) memcpy(all.data(), h, bytes);
    if (err) *err = *reinterpret_cast<int *>(p->h_red);
    *out = all[0];
    for (int s = 1; s < ns; ++s) {
        out->nan |= all[s].nan;
        out->iters_max = std::max(out->iters_max, all[s].iters_max);
        out->eta_max = std::max(out->eta_max, all[s].eta_max);
        out->iters += all[s].iters;
    }
    return KORE_OK;
}

// ---------------------------------------------------------------------------------
// Allocation-free solve: kore_solve_dev_noalloc (include/kore_gpu.h).
//
// Some callers cannot allocate device memory at the moment they need a solve: code
// that runs under a fixed memory budget or a pool it does not own, code that must not
// trigger the implicit device synchronisation of cudaMalloc/cudaFree inside a
// latency-critical loop, or a host library that is handed only a stream.  For them the
// scratch of one solve (padded right-hand side and solution, the reduction vectors of
// the sweep, the FP64 residual and the per-CTA maxima of the refinement loop, the
// norm partials, the refinement state and the error flag) lives in the file-scope array
// below instead of in buffers of the plan or of a caller.  Its size is fixed at kNoAllocMaxNp padded unknowns (about 2 MB, held by every GPU that
// loads the library until the process exits); larger problems are rejected.
// The kernels are the ones of kore_solve_dev; only their scratch pointers differ.
namespace {

constexpr int64_t kNoAllocMaxNp = 16384;
// stages x blocks of a sweep, (3 levels + 2) x blocks: a limit of the entry point, not of the
// scratch, which grows with the unknowns alone
constexpr int64_t kNoAllocMaxCnt = 32768;
constexpr int64_t kNoAllocMaxSpmvCta = (kNoAllocMaxNp * kRowLanes + 255) / 256 + kNoAllocMaxNp / 8 + 1;

struct NoAllocScratch {
    double2 bp[kNoAllocMaxNp];      // padded right-hand side (complex128)
    double2 xp[kNoAllocMaxNp];      // padded solution
    double2 r[kNoAllocMaxNp];       // FP64 residual of the refinement loop
    // sweep vectors, room for complex128: z, x, g and the levels' f, which take fewer than
    // blocks + levels blocks (20480 entries hold those of 16384 unknowns: at most 4 blocks of
    // 1024 more than the blocks themselves)
    double2 vecs[3 * kNoAllocMaxNp + 20480];
    double part[2 * kNoAllocMaxSpmvCta];   // per-CTA maxima of the residual kernel
    double red[2048 + 8];                  // ||b||_inf partials [0, 2048), then scalars
    IrState ir;
    int err;
    unsigned tick;
};

static __device__ __align__(256) NoAllocScratch g_noalloc_scratch;

// Device address of g_noalloc_scratch, looked up once per device (the symbol's name
// in host code is only a stand-in and must never be passed to a kernel).
std::mutex g_noalloc_mu;
NoAllocScratch *g_noalloc_addr[64] = {};

int noalloc_scratch(int device, NoAllocScratch **out) {
    if (device < 0 || device >= 64) return KORE_EINVAL;
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_addr[device]) {
        void *ptr = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
        if (e != cudaSuccess || !ptr) {
            std::fprintf(stderr, "kore: cudaGetSymbolAddress of the no-allocation scratch failed: %s\n",
                         cudaGetErrorString(e));
            return KORE_ECUDA;
        }
        g_noalloc_addr[device] = static_cast<NoAllocScratch *>(ptr);
    }
    *out = g_noalloc_addr[device];
    return KORE_OK;
}

// The launch is prepared per call, not kept in the plan: calls with scratches of their own
// may come from several threads.
template <typename C>
int noalloc_solve(kore_plan *p, NoAllocScratch *s, const double2 *b_dev, double2 *x_dev, double tol, cudaStream_t st) {
    const bool mixed = p->prec == KORE_PREC_MIXED;
    double *bn = s->red + 2048, *rn = s->red + 2049;
    SweepLaunch l;
    KORE_TRY(prepare_sweep<C>(p, p->sweep_cps > 0 ? TmaVariant{p->sweep_cps, p->sweep_chunk} : kTmaDefault, 1, l));
    SweepArgs a = sweep_args(p, 1);   // shift 0
    a.b = s->bp; a.bnorm = bn;
    a.vecs = s->vecs;
    a.out = s->xp; a.accumulate = 0; a.err = &s->err;
    a.skip = nullptr; a.skip_stride = 0; a.count = &s->ir.sweeps; a.count_total = &s->ir.sweeps_total;
    // every call starts from a cleared error flag, tick and refinement state
    KORE_CUDA_TRY(cudaMemsetAsync(&s->err, 0, 2 * sizeof(int), st));
    KORE_CUDA_TRY(cudaMemsetAsync(&s->ir, 0, sizeof(IrState), st));
    k_gather<<<std::min<unsigned>(kore_div_up(p->np, 256), 2048u), 256, 0, st>>>(p->np, p->n, p->d_slot2orig, b_dev,
                                                                                 s->bp);
    k_begin<<<kore_div_up(p->np, 256), 256, 0, st>>>(p->np, s->bp, s->red, bn, &s->tick, s->vecs, vec_bytes(p),
                                                     mixed ? &s->ir : nullptr, ~0u);
    KORE_LAUNCHED(2);
    KORE_TRY(launch_prepared<C>(l, a, p->num_sms, st));
    if (mixed) {
        const unsigned grid = spmv_grid(p);
        SpmvArgs ra = spmv_args(p, 2, s->xp, s->r);
        ra.lam = mk(p->sigma_re, p->sigma_im); ra.rhs = s->bp; ra.part = s->part; ra.skip = &s->ir.done;
        IrCheck chk{};
        chk.ir = &s->ir; chk.bnorm = bn; chk.minf = p->d_minf; chk.rn = rn; chk.tol = tol > 0.0 ? tol : 1e-14;
        chk.tick = &s->tick; chk.vecs = s->vecs; chk.vbytes = vec_bytes(p);
        a.b = s->r; a.bnorm = rn; a.accumulate = 1; a.skip = &s->ir.done;
        for (int it = 0; it < kIrMax; ++it) {
            k_spmv<<<grid, 256, spmv_smem(p), st>>>(ra, chk);
            KORE_LAUNCHED(1);
            KORE_TRY(launch_prepared<C>(l, a, p->num_sms, st));
        }
    }
    k_scatter<<<std::min<unsigned>(kore_div_up(p->np, 256), 2048u), 256, 0, st>>>(p->np, p->n, p->d_slot2orig, s->xp,
                                                                                  x_dev);
    KORE_LAUNCHED(1);
    KORE_CUDA_TRY(cudaGetLastError());
    return KORE_OK;
}

}  // namespace

extern "C" int kore_solve_dev_noalloc(kore_plan *p, const void *b_dev, void *x_dev, double refine_tol, void *stream) {
    if (!p || !b_dev || !x_dev) return KORE_EINVAL;
    if (p->np > kNoAllocMaxNp || (int64_t)(p->nlev > 0 ? 3 * p->nlev + 2 : 1) * p->K > kNoAllocMaxCnt) {
        std::fprintf(stderr,
                     "kore_solve_dev_noalloc: %lld padded unknowns in %d blocks exceed the fixed scratch "
                     "(%lld unknowns, %lld stages x blocks); use kore_solve_dev\n",
                     (long long)p->np, p->K, (long long)kNoAllocMaxNp, (long long)kNoAllocMaxCnt);
        return KORE_EINVAL;
    }
    if (!p->factored) return KORE_ENOTFACTORED;
    if (p->nshift != 1) {
        std::fprintf(stderr, "kore_solve_dev_noalloc: the plan holds %d factorised shifts; this entry point "
                             "solves with a plan of one shift (kore_factor)\n", p->nshift);
        return KORE_EINVAL;
    }
    int prev = -1;
    cudaGetDevice(&prev);
    if (prev != p->device) KORE_CUDA_TRY(cudaSetDevice(p->device));
    NoAllocScratch *s = nullptr;
    int rc = noalloc_scratch(p->device, &s);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const double2 *b = static_cast<const double2 *>(b_dev);
    double2 *x = static_cast<double2 *>(x_dev);
    if (rc == KORE_OK)
        rc = p->prec == KORE_PREC_MIXED ? noalloc_solve<float2>(p, s, b, x, refine_tol, st)
                                        : noalloc_solve<double2>(p, s, b, x, refine_tol, st);
    if (rc == KORE_OK) {
        // wait for this call's kernels, then read its error flag and NaN state
        int flags[2] = {0, 0};
        if (cudaMemcpyAsync(&flags[0], &s->err, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaMemcpyAsync(&flags[1], &s->ir.nan, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess)
            rc = KORE_ECUDA;
        else if (flags[0] != 0)
            rc = KORE_ETIMEOUT;
        else if (flags[1] != 0)
            rc = KORE_ENAN;
    }
    if (prev >= 0 && prev != p->device) cudaSetDevice(prev);
    return rc;
}
