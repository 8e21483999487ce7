// Complex64 GEMMs of the mixed-precision factorisation on the 5th-generation tensor
// cores (tcgen05), in three-pass TF32 (3xTF32):
//     x = x_hi + x_lo,  x_hi = x rounded to TF32,  x_lo = x - x_hi (exact in FP32),
//     a b ~ a_hi b_hi + a_hi b_lo + a_lo b_hi      (FP32 accumulation in tensor memory)
// and each complex product as four real ones,
//     Re(AB) = Ar Br - Ai Bi,  Im(AB) = Ar Bi + Ai Br
// (the MMA's negate bit makes the subtraction).
//
// Data flow of one 128 x 128 tile of C = beta C + alpha (A1 B1 [+ A2 B2]), one CTA:
//   * the operands are split inside the kernel, 32 columns of K at a time: four warps load
//     the 128 rows of A (one thread per row, coalesced along the column-major rows) and
//     write the planes Re hi, Re lo, Im hi, Im lo to tensor memory, where the MMA takes
//     its A operand from; four warps load the columns of B (K contiguous) and write the
//     same four planes to shared memory in the 128-byte swizzled K-major layout;
//   * each of the two stages has a "full" mbarrier (one arrival per converting warp) and an
//     "empty" one (tcgen05.commit); the next slice's loads are in flight while a stage waits;
//   * one thread issues tcgen05.mma (M = 128, N up to 128, K = 8, twelve per step of K) into
//     the tensor-memory accumulators Re (columns 0-127) and Im (128-255);
//   * the eight converting warps read the accumulators back with tcgen05.ld and write C.
// What bounds it: the MMAs (a 32-wide slice takes 48 of them, about 3,070 cycles).  Both
// operands from shared memory kept it at the shared-memory bandwidth (8 KB per MMA of 64
// cycles, plus the copies), and planes split beforehand by another kernel made the copies
// 2.3 times the operands: with A in tensor memory and the split in the kernel a slice
// moves 64 KB from L2 per 3,070 cycles and shared memory serves B alone.  (59 products of
// S = 240, 236 tiles: the tensor pipe is busy for 57% of the SMs' active cycles, 52% with an
// accumulated C; 40 and 37% of the launch, whose second wave is half empty.)
// Every wait is bounded (error flag, then the kernel carries on to release its tensor
// memory); tensor memory is allocated and freed by warp 8.
#include "kore_internal.cuh"
#include "kore_tma.cuh"
#include <algorithm>
#include <cstdio>
#include <vector>

namespace {

// A 128 x 64 tile with one stage and two CTAs per SM, meant to overlap one CTA's epilogue
// with the other's MMAs, took 2.5 times as long: each slice then waits for its conversion.
constexpr int kTcM = 128, kTcN = 128, kTcK = 32, kTcStages = 2;
constexpr int kTcConvWarps = 8;                   // 4 for A, 4 for B; warp 8 issues the MMAs
constexpr int kTcThreads = 32 * (kTcConvWarps + 1);
constexpr int kPlanes = 4;                        // Re hi, Re lo, Im hi, Im lo
constexpr int kPlaneB = kTcN * kTcK * 4;          // 16 KB: one plane of a B slice
constexpr int kStageB = kPlanes * kPlaneB;
// tensor memory: Re and Im accumulators, then the A planes (32 columns each) of the stages
constexpr uint32_t kTmemA = 2 * kTcN;
constexpr uint32_t kTmemCols = kTmemA + kTcStages * kPlanes * kTcK;   // 512, all of it
// more than half of an SM's shared memory, so that no second CTA waits there for tensor memory
constexpr size_t kTcSmem = (size_t)kTcStages * kStageB + 1024 + 128;
static_assert(kTmemCols == 512 && 2 * kTcSmem > 227 * 1024, "one CTA per SM");

struct TcJob {
    const float2 *A1, *B1, *A2, *B2;   // column-major S x S (A2 null: one product)
    float2 *C;                         // column-major S x S
    float alpha;                       // C = beta C + alpha (A1 B1 + A2 B2)
    int beta;
};

struct TcParams {
    const TcJob *jobs;
    int S, tiles_n;
    int *err;
};

// ----------------------------------------------------------------------------- tcgen05 PTX
__device__ __forceinline__ void tc_alloc(uint32_t *holder, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(holder)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// D[tmem] (+)= A[tmem] B[smem]; accumulate = 0 overwrites D
__device__ __forceinline__ void tc_mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
        "r"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}

// arrive on `bar` once every MMA this thread issued before has completed
__device__ __forceinline__ void tc_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// 16 consecutive 32-bit columns of this warp's 32 lanes
__device__ __forceinline__ void tc_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
// write 16 consecutive 32-bit columns of this warp's 32 lanes
__device__ __forceinline__ void tc_st16(uint32_t taddr, const float (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};" ::"f"(v[0]),
        "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "f"(v[8]), "f"(v[9]),
        "f"(v[10]), "f"(v[11]), "f"(v[12]), "f"(v[13]), "f"(v[14]), "f"(v[15]), "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tc_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// generic-proxy writes to shared memory visible to the MMA (async proxy)
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor of a K-major operand in the 128-byte swizzled layout:
// rows of 128 bytes (32 TF32 of K), 8-row groups 1024 bytes apart.
//   [0,14) start address >> 4, [16,30) leading byte offset >> 4 (unused here: 1),
//   [32,46) stride byte offset >> 4 = 1024 >> 4, [46,48) version 1,
//   [49,52) base offset 0 (1024-byte aligned tiles), [61,64) layout 2 = 128-byte swizzle.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
    return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

// Instruction descriptor of kind::tf32: D F32 (bits 4-5 = 1), A and B TF32 (bits 7-9,
// 10-12 = 2), A negated (bit 13), both operands K-major (bits 15, 16 = 0), N >> 3 at bits
// 17-22, M >> 4 at bits 24-28.
__device__ __forceinline__ uint32_t tf32_idesc(int n, int negate_a) {
    return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)negate_a << 13) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(kTcM >> 4) << 24);
}

__device__ __forceinline__ float tf32_rna(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return __uint_as_float(r);
}

// ----------------------------------------------------------------------------- GEMM
__global__ void __launch_bounds__(kTcThreads, 1) k_tc_gemm(const TcParams P) {
    extern __shared__ unsigned char smem_raw[];
    // 1024-byte aligned stages (the 128-byte swizzle pattern repeats every 1024 bytes)
    unsigned char *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + kTcStages * kStageB);
    uint64_t *empty = full + kTcStages;
    uint64_t *accum = empty + kTcStages;
    uint32_t *holder = reinterpret_cast<uint32_t *>(accum + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const TcJob job = P.jobs[blockIdx.y];
    const int S = P.S;
    const int tm = blockIdx.x / P.tiles_n, tn = blockIdx.x - tm * P.tiles_n;
    const int nk = (S + kTcK - 1) / kTcK;
    const int nstage = (job.A2 ? 2 : 1) * nk;
    const int m0 = tm * kTcM, n0 = tn * kTcN;
    const int n_eff = min(kTcN, (S - n0 + 15) & ~15);   // columns the MMAs compute
    if (tid == 0) {
        for (int s = 0; s < kTcStages; ++s) {
            mbar_init(&full[s], kTcConvWarps);
            mbar_init(&empty[s], 1);
        }
        mbar_init(accum, 1);
        mbar_fence_init();
    }
    if (warp == kTcConvWarps) tc_alloc(holder, kTmemCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *holder;

    if (warp < 4) {
        // A: thread = row, its 32 entries of the slice in registers, planes to tensor memory
        const int row = m0 + warp * 32 + lane;
        float2 v[kTcK];
        auto load = [&](int ks) {
            const float2 *A = (ks >= nk ? job.A2 : job.A1) + row;
            const int k0 = (ks >= nk ? ks - nk : ks) * kTcK;
#pragma unroll
            for (int k = 0; k < kTcK; ++k)
                v[k] = (row < S && k0 + k < S) ? __ldg(A + (int64_t)(k0 + k) * S) : make_float2(0.f, 0.f);
        };
        load(0);
        for (int ks = 0; ks < nstage; ++ks) {
            const int s = ks % kTcStages;
            if (!mbar_wait(&empty[s], ((uint32_t)(ks / kTcStages) & 1u) ^ 1u)) atomicCAS(P.err, 0, KORE_DEVERR_FLAG);
            tc_fence_after();
            const uint32_t ta = tmem + kTmemA + (uint32_t)(s * kPlanes * kTcK) + ((uint32_t)(warp * 32) << 16);
#pragma unroll
            for (int p = 0; p < kPlanes; ++p)
#pragma unroll
                for (int h = 0; h < kTcK; h += 16) {
                    float r[16];
#pragma unroll
                    for (int k = 0; k < 16; ++k) {
                        const float x = p < 2 ? v[h + k].x : v[h + k].y, hi = tf32_rna(x);
                        r[k] = (p & 1) ? x - hi : hi;
                    }
                    tc_st16(ta + (uint32_t)(p * kTcK + h), r);
                }
            if (ks + 1 < nstage) load(ks + 1);
            tc_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
        }
    } else if (warp < kTcConvWarps) {
        // B: thread = four entries of K (chunk ch) of columns n, n + 16, ..., planes to shared
        // memory: row n of a plane is 128 bytes of K, its 16-byte chunk ch at ch ^ (n & 7)
        const int ch = lane & 7, nb = (warp - 4) * 4 + (lane >> 3);
        const bool vec = (S & 3) == 0;   // every column starts on a 32-byte boundary
        float4 v[kTcN / 16][2];
        auto load = [&](int ks) {
            const float2 *B = ks >= nk ? job.B2 : job.B1;
            const int k0 = (ks >= nk ? ks - nk : ks) * kTcK + 4 * ch;
#pragma unroll
            for (int i = 0; i < kTcN / 16; ++i) {
                const int n = n0 + nb + 16 * i;
                v[i][0] = v[i][1] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (n < S && k0 < S) {
                    const float2 *b = B + (int64_t)n * S + k0;
                    if (vec) {
                        v[i][0] = __ldg(reinterpret_cast<const float4 *>(b));
                        v[i][1] = __ldg(reinterpret_cast<const float4 *>(b) + 1);
                    } else {
                        const float2 z = make_float2(0.f, 0.f);
                        const float2 b0 = b[0], b1 = k0 + 1 < S ? b[1] : z, b2 = k0 + 2 < S ? b[2] : z,
                                     b3 = k0 + 3 < S ? b[3] : z;
                        v[i][0] = make_float4(b0.x, b0.y, b1.x, b1.y);
                        v[i][1] = make_float4(b2.x, b2.y, b3.x, b3.y);
                    }
                }
            }
        };
        load(0);
        for (int ks = 0; ks < nstage; ++ks) {
            const int s = ks % kTcStages;
            if (!mbar_wait(&empty[s], ((uint32_t)(ks / kTcStages) & 1u) ^ 1u)) atomicCAS(P.err, 0, KORE_DEVERR_FLAG);
            unsigned char *sb = smem + (size_t)s * kStageB;
#pragma unroll
            for (int i = 0; i < kTcN / 16; ++i) {
                const int n = nb + 16 * i;
                if (n >= n_eff) continue;
                float4 *d = reinterpret_cast<float4 *>(sb + n * 128 + ((ch ^ (n & 7)) << 4));
                const float4 re = make_float4(v[i][0].x, v[i][0].z, v[i][1].x, v[i][1].z);
                const float4 im = make_float4(v[i][0].y, v[i][0].w, v[i][1].y, v[i][1].w);
                const float4 rh = make_float4(tf32_rna(re.x), tf32_rna(re.y), tf32_rna(re.z), tf32_rna(re.w));
                const float4 ih = make_float4(tf32_rna(im.x), tf32_rna(im.y), tf32_rna(im.z), tf32_rna(im.w));
                d[0] = rh;
                d[1 * kPlaneB / 16] = make_float4(re.x - rh.x, re.y - rh.y, re.z - rh.z, re.w - rh.w);
                d[2 * kPlaneB / 16] = ih;
                d[3 * kPlaneB / 16] = make_float4(im.x - ih.x, im.y - ih.y, im.z - ih.z, im.w - ih.w);
            }
            if (ks + 1 < nstage) load(ks + 1);
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
        }
    } else if (lane == 0) {
        // MMA issuer
        const uint32_t ip = tf32_idesc(n_eff, 0), in = tf32_idesc(n_eff, 1);
        const uint32_t re = tmem, im = tmem + kTcN;
        for (int ks = 0; ks < nstage; ++ks) {
            const int s = ks % kTcStages;
            if (!mbar_wait(&full[s], (uint32_t)(ks / kTcStages) & 1u)) atomicCAS(P.err, 0, KORE_DEVERR_FLAG);
            tc_fence_after();
            const uint32_t ta = tmem + kTmemA + (uint32_t)(s * kPlanes * kTcK);
            const uint32_t sb = smem_u32(smem + (size_t)s * kStageB);
#pragma unroll
            for (int k8 = 0; k8 < kTcK / 8; ++k8) {
                uint32_t a[kPlanes];
                uint64_t b[kPlanes];
#pragma unroll
                for (int p = 0; p < kPlanes; ++p) {
                    a[p] = ta + (uint32_t)(p * kTcK + 8 * k8);
                    b[p] = sw128_desc(sb + p * kPlaneB) + (uint64_t)(2 * k8);   // + 32 bytes of K
                }
                const uint32_t acc = (ks == 0 && k8 == 0) ? 0u : 1u;
                // Re += Ar Br - Ai Bi, Im += Ar Bi + Ai Br; hi hi, hi lo, lo hi of each
                tc_mma_ts(re, a[0], b[0], ip, acc);
                tc_mma_ts(im, a[0], b[2], ip, acc);
                tc_mma_ts(re, a[0], b[1], ip, 1u);
                tc_mma_ts(im, a[0], b[3], ip, 1u);
                tc_mma_ts(re, a[1], b[0], ip, 1u);
                tc_mma_ts(im, a[1], b[2], ip, 1u);
                tc_mma_ts(re, a[2], b[2], in, 1u);
                tc_mma_ts(im, a[2], b[0], ip, 1u);
                tc_mma_ts(re, a[2], b[3], in, 1u);
                tc_mma_ts(im, a[2], b[1], ip, 1u);
                tc_mma_ts(re, a[3], b[2], in, 1u);
                tc_mma_ts(im, a[3], b[0], ip, 1u);
            }
            tc_commit(&empty[s]);   // the stage is free once these MMAs have read it
        }
        tc_commit(accum);
    }
    __syncwarp();

    // epilogue: converting warp w reads rows 32 (w % 4) .. + 31 (the tensor-memory lanes it
    // can reach) of columns 64 (w / 4) .. + 63
    if (warp < kTcConvWarps) {
        if (!mbar_wait(accum, 0)) atomicCAS(P.err, 0, KORE_DEVERR_FLAG);
        tc_fence_after();
        const int row = m0 + (warp & 3) * 32 + lane;
        const uint32_t tl = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        const int cb = (warp >> 2) * (kTcN / 2);
#pragma unroll
        for (int c0 = cb; c0 < cb + kTcN / 2; c0 += 16) {
            if (c0 >= n_eff) break;
            // C's old entries are loaded together, ahead of the stores they must not wait for
            float2 o[16];
            float2 *c = job.C + row + (int64_t)(n0 + c0) * S;
#pragma unroll
            for (int j = 0; j < 16; ++j)
                o[j] = (job.beta && row < S && n0 + c0 + j < S) ? c[(int64_t)j * S] : make_float2(0.f, 0.f);
            float re[16], im[16];
            tc_ld16(tl + (uint32_t)c0, re);
            tc_ld16(tl + (uint32_t)(kTcN + c0), im);
            tc_ld_wait();
            if (row < S) {
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    if (n0 + c0 + j < S) {
                        float2 v = make_float2(job.alpha * re[j], job.alpha * im[j]);
                        if (job.beta) {
                            v.x += o[j].x;
                            v.y += o[j].y;
                        }
                        c[(int64_t)j * S] = v;
                    }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kTcConvWarps) tc_dealloc(tmem, kTmemCols);
}

// ----------------------------------------------------------------------------- host
// Runs the jobs (device array of njobs).  No job may read what another of the same call
// writes.
int tc_run(cudaStream_t st, int device, int S, const TcJob *jobs, int njobs, int *err) {
    if (njobs == 0) return KORE_OK;
    TcParams P;
    P.S = S;
    P.tiles_n = kore_div_up(S, kTcN);
    P.err = err;
    const int tiles = kore_div_up(S, kTcM) * P.tiles_n;
    KORE_TRY(kore_allow_max_dyn_smem(k_tc_gemm, device));
    for (int j0 = 0; j0 < njobs; j0 += 65535) {
        P.jobs = jobs + j0;
        k_tc_gemm<<<dim3(tiles, std::min(65535, njobs - j0)), kTcThreads, kTcSmem, st>>>(P);
        KORE_LAUNCHED(1);
    }
    KORE_CUDA_TRY(cudaGetLastError());
    return KORE_OK;
}

// FP64 reference of the self-test: C_ref(r, c) = beta C0 + alpha sum of the products
// and the magnitude bound sum |a| |b| (one thread per element).
__global__ void k_tc_ref(int S, const TcJob *jobs, int njobs, const float2 *C0, double *err) {
    const int j = blockIdx.y;
    if (j >= njobs) return;
    const TcJob jb = jobs[j];
    const int64_t SS = (int64_t)S * S;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < SS; e += (int64_t)gridDim.x * blockDim.x) {
        const int r = (int)(e % S), c = (int)(e / S);
        double sr = 0, si = 0, mag = 0;
        for (int pr = 0; pr < 2; ++pr) {
            const float2 *A = pr ? jb.A2 : jb.A1, *B = pr ? jb.B2 : jb.B1;
            if (!A) continue;
            for (int k = 0; k < S; ++k) {
                const float2 a = A[r + (int64_t)k * S], b = B[k + (int64_t)c * S];
                sr += (double)a.x * b.x - (double)a.y * b.y;
                si += (double)a.x * b.y + (double)a.y * b.x;
                mag += (fabs((double)a.x) + fabs((double)a.y)) * (fabs((double)b.x) + fabs((double)b.y));
            }
        }
        double rr = jb.alpha * sr, ri = jb.alpha * si;
        if (jb.beta) { rr += C0[j * SS + e].x; ri += C0[j * SS + e].y; }
        const float2 got = jb.C[e];
        const double d = fmax(fabs(got.x - rr), fabs(got.y - ri)) / fmax(mag, 1e-30);
        // max of non-negative doubles through their bit patterns
        atomicMax(reinterpret_cast<unsigned long long *>(err), (unsigned long long)__double_as_longlong(d));
    }
}

__global__ void k_tc_fill(float2 *x, int64_t n, uint64_t seed) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        uint64_t h = (uint64_t)i * 0x9E3779B97F4A7C15ULL + seed;
        h ^= h >> 31; h *= 0xBF58476D1CE4E5B9ULL; h ^= h >> 27; h *= 0x94D049BB133111EBULL; h ^= h >> 31;
        const float u = (float)(h & 0xFFFFFF) / 16777216.f - 0.5f;
        const float v = (float)((h >> 24) & 0xFFFFFF) / 16777216.f - 0.5f;
        x[i] = make_float2(u, v);
    }
}

}  // namespace

// ----------------------------------------------------------------------------- factorisation use
// Bytes of the job table for one reduction level of `cap` shifts; the plan allocates the
// largest over its levels.
int64_t kore_tc_table_bytes(const kore_plan *p, int cap) {
    int64_t nj = 0;
    for (int l = 0; l < p->nlev; ++l)
        // even update (levels >= 1): 3 neven jobs; G, H and their refinement: 2 nodd jobs
        nj = std::max<int64_t>(nj, std::max(l > 0 ? 3 * p->lev[l].neven : 0, 2 * p->lev[l].nodd));
    return nj * cap * (int64_t)sizeof(TcJob) + 64;
}

static int tc_upload_run(kore_plan *p, const std::vector<TcJob> &jobs) {
    KORE_CUDA_TRY(cudaMemcpyAsync(p->d_tctab, jobs.data(), jobs.size() * sizeof(TcJob), cudaMemcpyHostToDevice,
                                  p->stream));
    return tc_run(p->stream, p->device, p->S, static_cast<const TcJob *>(p->d_tctab), (int)jobs.size(), p->d_err);
}

// Even-block update of level l >= 1 for every shift (complex64 factors):
// D_i -= L_q H_jl + U_q G_jr;  L' = -L_q G_jl;  U' = -U_q H_jr.
int kore_even_update_tc(kore_plan *p, const BcrLevel &lv) {
    const int S = p->S, ns = p->fw_n;
    const int64_t lo = p->fw_lo;   // shift sh of the factor window is shift lo + sh of the plan
    const int64_t SS = (int64_t)S * S;
    std::vector<TcJob> jobs;
    for (int sh = 0; sh < ns; ++sh) {
        float2 *LU = static_cast<float2 *>(p->d_LU) + (lo + sh) * p->lu_stride();
        float2 *Dw = static_cast<float2 *>(p->d_Dw) + (lo + sh) * p->f_stride();
        const float2 *G = static_cast<const float2 *>(p->d_Gm) + (lo + sh) * p->f_stride();
        const float2 *H = static_cast<const float2 *>(p->d_Hm) + (lo + sh) * p->f_stride();
        for (int e = 0; e < lv.neven; ++e) {
            const int64_t q = 2 * e, jl = (q - 1) * lv.stride * SS, jr = (q + 1) * lv.stride * SS;
            const bool hasl = q >= 1, hasr = q + 1 < lv.Kl;
            const float2 *Lq = LU + (lv.lu_L + q) * SS, *Uq = LU + (lv.lu_U + q) * SS;
            float2 *D = Dw + q * lv.stride * SS;
            if (hasl && hasr) jobs.push_back(TcJob{Lq, H + jl, Uq, G + jr, D, -1.f, 1});
            else if (hasl) jobs.push_back(TcJob{Lq, H + jl, nullptr, nullptr, D, -1.f, 1});
            else if (hasr) jobs.push_back(TcJob{Uq, G + jr, nullptr, nullptr, D, -1.f, 1});
            if (lv.lu_nL >= 0 && q >= 2)
                jobs.push_back(TcJob{Lq, G + jl, nullptr, nullptr, LU + (lv.lu_nL + e) * SS, -1.f, 0});
            if (lv.lu_nU >= 0 && q + 2 < lv.Kl)
                jobs.push_back(TcJob{Uq, H + jr, nullptr, nullptr, LU + (lv.lu_nU + e) * SS, -1.f, 0});
        }
    }
    return tc_upload_run(p, jobs);
}

// R(k, c) += rs_k a_e for the level-0 couplings of the odd blocks (side 0: L_j into
// R_G, side 1: U_j into R_H), R_G and R_H at Rbase + shift * t_stride + o * 2 S^2 (+ S^2).
// CTA = (odd index o, side, shift); threads over the columns.
__global__ void k_add_couplings(const int *__restrict__ cc_ptr, const int *__restrict__ cc_row,
                                const int *__restrict__ cc_src, const double2 *__restrict__ aval,
                                const double *__restrict__ rscale, int S, int64_t np, float2 *Rbase,
                                int64_t t_stride) {
    const int64_t o = blockIdx.x, side = blockIdx.y, sh = blockIdx.z;
    const int64_t SS = (int64_t)S * S, j = 2 * o + 1;
    const int *ptr = cc_ptr + (2 * o + side) * (int64_t)(S + 1);
    const double *rs = rscale + sh * np + j * S;
    float2 *R = Rbase + sh * t_stride + o * 2 * SS + side * SS;
    for (int c = threadIdx.x; c < S; c += blockDim.x)
        for (int t = ptr[c]; t < ptr[c + 1]; ++t) {
            const int k = cc_row[t];
            const double2 a = rs[k] * aval[cc_src[t]];
            float2 &r = R[k + (int64_t)c * S];
            r = make_float2((float)((double)r.x + a.x), (float)((double)r.y + a.y));
        }
}

// G_j = D_j^-1 L_j and H_j = D_j^-1 U_j of the odd blocks of a level for every shift
// (complex64 factors), on the tensor cores, with one step of refinement:
//     G0 = D^-1 L,   R = L - D G0,   G = G0 + D^-1 R
// (D is the row-scaled diagonal block, D^-1 its Gauss-Jordan inverse).  The product with
// an explicit inverse loses accuracy where D^-1 L cancels; the refinement step gives
// the columns of G the accuracy of a stable solve, which keeps the FP64 refinement of
// the solves at two to three corrections.  Level >= 1: dense L, U in the coupling
// store (the odd blocks' L, U are not read again, so R overwrites them).  Level 0:
// G0 and H0 come from the sparse couplings (k_gh_l0); R goes to the Gauss-Jordan work
// area T, free after the extraction.
int kore_gh_update_tc(kore_plan *p, const BcrLevel &lv, int level0) {
    const int S = p->S, ns = p->fw_n;
    const int64_t lo = p->fw_lo;   // shift sh of the factor window is shift lo + sh of the plan
    const int64_t SS = (int64_t)S * S, no = lv.nodd;
    float2 *Dinv = static_cast<float2 *>(p->d_Dinv), *Dw = static_cast<float2 *>(p->d_Dw);
    float2 *G = static_cast<float2 *>(p->d_Gm), *H = static_cast<float2 *>(p->d_Hm);
    float2 *LU = static_cast<float2 *>(p->d_LU), *T = static_cast<float2 *>(p->d_T);
    auto blk = [&](float2 *base, int sh, int64_t o) {
        return base + (lo + sh) * p->f_stride() + (2 * o + 1) * lv.stride * SS;
    };
    // residual storage of (shift, odd o, side)
    auto rstore = [&](int sh, int64_t o, int side) -> float2 * {
        if (level0) return T + (lo + sh) * p->t_stride() + o * 2 * SS + side * SS;
        return LU + (lo + sh) * p->lu_stride() + ((side ? lv.lu_U : lv.lu_L) + 2 * o + 1) * SS;
    };
    auto hasr = [&](int64_t o) { return 2 * o + 2 < lv.Kl; };
    // one job per (shift, odd block, side): C = beta C + alpha A B with A the block's matrix
    std::vector<TcJob> jobs;
    auto run = [&](float2 *A, auto B, auto Cm, float alpha, int beta) {
        jobs.clear();
        for (int sh = 0; sh < ns; ++sh)
            for (int64_t o = 0; o < no; ++o) {
                jobs.push_back(TcJob{blk(A, sh, o), B(sh, o, 0), nullptr, nullptr, Cm(sh, o, 0), alpha, beta});
                if (hasr(o)) jobs.push_back(TcJob{blk(A, sh, o), B(sh, o, 1), nullptr, nullptr, Cm(sh, o, 1), alpha, beta});
            }
        return tc_upload_run(p, jobs);
    };
    auto gh = [&](int sh, int64_t o, int side) { return blk(side ? H : G, sh, o); };
    // levels >= 1: G0 = D^-1 L, H0 = D^-1 U
    if (!level0) KORE_TRY(run(Dinv, rstore, gh, 1.f, 0));
    // R = L - D G0 (level 0: R = -D G0, then + L from the sparse couplings)
    KORE_TRY(run(Dw, gh, rstore, -1.f, level0 ? 0 : 1));
    if (level0) {
        k_add_couplings<<<dim3((unsigned)no, 2, ns), 256, 0, p->stream>>>(p->d_cc_ptr, p->d_cc_row, p->d_cc_src,
                                                                          p->d_aval, p->d_rscale + lo * p->np, S,
                                                                          p->np, T + lo * p->t_stride(),
                                                                          p->t_stride());
        KORE_LAUNCHED(1);
    }
    // G = G0 + D^-1 R
    return run(Dinv, rstore, gh, 1.f, 1);
}

extern "C" int kore_tc_selftest(int device, int S, int nmat, double *max_rel_err) {
    if (!max_rel_err || S <= 0 || S > 1024 || nmat < 2 || nmat > 64) return KORE_EINVAL;
    int prev = -1;
    cudaGetDevice(&prev);
    KORE_CUDA_TRY(cudaSetDevice(device));
    const int64_t SS = (int64_t)S * S;
    float2 *A = nullptr, *B = nullptr, *C = nullptr, *C0 = nullptr;
    TcJob *tab = nullptr;
    double *err = nullptr;
    int *flag = nullptr;
    int rc = KORE_OK;
    auto ck = [&](cudaError_t e) { if (e != cudaSuccess && rc == KORE_OK) rc = (e == cudaErrorMemoryAllocation) ? KORE_ENOMEM : KORE_ECUDA; };
    ck(cudaMalloc(&A, nmat * SS * sizeof(float2)));
    ck(cudaMalloc(&B, nmat * SS * sizeof(float2)));
    ck(cudaMalloc(&C, nmat * SS * sizeof(float2)));
    ck(cudaMalloc(&C0, nmat * SS * sizeof(float2)));
    ck(cudaMalloc(&tab, (size_t)nmat * sizeof(TcJob)));
    ck(cudaMalloc(&err, sizeof(double)));
    ck(cudaMalloc(&flag, sizeof(int)));
    if (rc == KORE_OK) {
        k_tc_fill<<<256, 256>>>(A, nmat * SS, 1);
        k_tc_fill<<<256, 256>>>(B, nmat * SS, 2);
        k_tc_fill<<<256, 256>>>(C, nmat * SS, 3);
        ck(cudaMemcpy(C0, C, nmat * SS * sizeof(float2), cudaMemcpyDeviceToDevice));
        ck(cudaMemset(err, 0, sizeof(double)));
        ck(cudaMemset(flag, 0, sizeof(int)));
        // job m: even m: C_m = A_m B_m;  odd m: C_m -= A_m B_m + A_{m-1} B_{m+1 mod n}
        std::vector<TcJob> jobs;
        for (int m = 0; m < nmat; ++m) {
            if (m % 2 == 0) jobs.push_back(TcJob{A + m * SS, B + m * SS, nullptr, nullptr, C + m * SS, 1.f, 0});
            else jobs.push_back(TcJob{A + m * SS, B + m * SS, A + (m - 1) * SS, B + (m + 1) % nmat * SS, C + m * SS, -1.f, 1});
        }
        ck(cudaMemcpy(tab, jobs.data(), jobs.size() * sizeof(TcJob), cudaMemcpyHostToDevice));
        if (rc == KORE_OK) rc = tc_run(0, device, S, tab, nmat, flag);
        if (rc == KORE_OK) {
            k_tc_ref<<<dim3(64, nmat), 256>>>(S, tab, nmat, C0, err);
            ck(cudaGetLastError());
            ck(cudaDeviceSynchronize());
            int h = 0;
            ck(cudaMemcpy(&h, flag, sizeof(int), cudaMemcpyDeviceToHost));
            ck(cudaMemcpy(max_rel_err, err, sizeof(double), cudaMemcpyDeviceToHost));
            if (rc == KORE_OK && h != 0) rc = KORE_ETIMEOUT;
        }
    }
    cudaFree(A); cudaFree(B); cudaFree(C); cudaFree(C0); cudaFree(tab); cudaFree(err); cudaFree(flag);
    if (prev >= 0) cudaSetDevice(prev);
    return rc;
}
