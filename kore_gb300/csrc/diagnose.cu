// Flow diagnostics of eigenvectors on the GPU: what bin/spin_doctor.py computes with
// bin/utils4pp.py (diagnose, flow_worker) for the hydrodynamic problem in a shell.
//
// For every degree l of a velocity eigenvector (poloidal coefficients P_l, toroidal
// T_l, N Chebyshev coefficients each, radius mapped to [ricb, rcmb]):
//   * the radial function and its r-derivatives at the N Chebyshev-Gauss points
//     x_i = cos((i + 1/2) pi / N) (bin/utils4pp.py:805-829, funcheb :28-51);
//   * the radial, consoidal and toroidal components q, s, t (cheb2space_pol/tor,
//     :163-218) and the integrands of the kinetic energy, of integral(u . lap u) and of
//     the internal dissipation (:221-296);
//   * their Chebyshev-Gauss quadratures (cg_quad, :54-64).
// The sums over l, the scaling by OmgTau Ek and the power-balance residuals
// (bin/spin_doctor.py:148-160, 225-236) are left to the caller (kore_gb300/diagnostics.py).
//
// Chebyshev polynomials and their derivatives are even or odd, d^j T_k(-x) =
// (-1)^(k+j) d^j T_k(x), and the points are symmetric, so a pair of points x, -x takes one
// pass over the coefficients: the sums over even and over odd k, added for x and subtracted
// for -x.  That is half of the FP64 products, whose pipe (two multiply-adds per SM per clock)
// bounds the kernel: 16 modes of the 240k-unknown shell took 19.2 ms with every point on its
// own, of which 17 ms at the pipe's rate.
// Layout: k_cheb_eval writes E[j][k][i] = d^j T_k / dr^j (x_i), j = 0..3, for the points
// i < nh = ceil(N / 2) with x_i >= 0 (threads over points, three-term recurrences of T_k and
// its r-derivatives), then x_i and the quadrature weights.  k_flow_integrals runs one CTA per
// (degree block, KV eigenvectors), the coefficients in shared memory; R threads share a pair
// of points, thread role r summing over k = r, r + R, ... (R even, so a role's k have one
// parity), and the three integrals are reduced in a fixed order.
#include "kore_internal.cuh"
#include <algorithm>
#include <vector>

namespace {

constexpr int kDiagThreads = 512;   // at most, roles x points

__global__ void k_cheb_eval(int N, double ricb, double rcmb, double *__restrict__ E) {
    const int nh = (N + 1) / 2;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nh) return;
    // the middle point of an odd N is 0 (cos(pi / 2) rounds to 6e-17)
    const double x = (2 * i + 1 == N) ? 0.0 : cos((i + 0.5) * 3.14159265358979323846 / N);
    const double dr = 2.0 / (rcmb - ricb);   // dx/dr
    const int64_t NN = (int64_t)N * nh;
    E[4 * NN + i] = x;
    E[4 * NN + nh + i] = sqrt(1.0 - x * x);
    // T_k and its first three r-derivatives: T_{k+1} = 2x T_k - T_{k-1} differentiated
    // (dx/dr = dr), seven FP64 operations per step
    const double x2 = 2.0 * x, c1 = 2.0 * dr, c2 = 4.0 * dr, c3 = 6.0 * dr;
    double t0 = 1.0, t1 = x;            // T_{k-1}, T_k
    double d10 = 0.0, d11 = dr;         // first derivative
    double d20 = 0.0, d21 = 0.0;        // second
    double d30 = 0.0, d31 = 0.0;        // third
    for (int k = 0; k < N; ++k) {       // (t0, d10, ...) belongs to k
        const int64_t at = (int64_t)k * nh + i;
        E[at] = t0;
        E[NN + at] = d10;
        E[2 * NN + at] = d20;
        E[3 * NN + at] = d30;
        const double n0 = fma(x2, t1, -t0);
        const double n1 = fma(c1, t1, fma(x2, d11, -d10));
        const double n2 = fma(c2, d11, fma(x2, d21, -d20));
        const double n3 = fma(c3, d21, fma(x2, d31, -d30));
        t0 = t1; t1 = n0; d10 = d11; d11 = n1; d20 = d21; d21 = n2; d30 = d31; d31 = n3;
    }
}

struct FlowArgs {
    int N, npol, ntor, nvec;
    double ricb, rcmb;
    const int *lpol, *ltor;      // degrees of the poloidal and toroidal blocks
    const double2 *x;            // nvec vectors of (npol + ntor) N complex coefficients:
    int64_t vstride, cstride;    // coefficient i of vector v at x[v vstride + i cstride]
    const double *E;             // evaluation matrices, points and weights (k_cheb_eval)
    double *out;                 // per (vector, block): energy, diffusion, internal dissipation
};

// Integrands (energy, diffusion, internal dissipation) at radius rk from the radial
// function and its derivatives p.
__device__ __forceinline__ void flow_integrands(bool tor, int l, double rk, const double2 (&p)[4], double (&f)[3]) {
    const double L = (double)l * (l + 1), f0 = 4.0 * 3.14159265358979323846 / (2 * l + 1);
    const double r2 = rk * rk;
    if (!tor) {
        const double ri = 1.0 / rk, li = 1.0 / L;
        const double2 q0 = (L / rk) * p[0];
        const double2 s0 = p[1] + ri * p[0];
        const double2 q1 = ri * (L * p[1] - q0);
        const double2 s1 = p[2] + li * q1;
        const double2 q2 = ri * (L * p[2] - 2.0 * q1);
        const double2 s2 = p[3] + li * q2;
        f[0] = f0 * (r2 * abs2(q0) + r2 * L * abs2(s0));
        const double2 t = L * r2 * (conjg(s0) * s2) + (2.0 * rk * L) * (conjg(s0) * s1) +
                          (-(L * L)) * (conjg(s0) * s0) + (-((double)l * l + l + 2)) * (conjg(q0) * q0) +
                          (2.0 * rk) * (conjg(q0) * q1) + r2 * (conjg(q0) * q2) +
                          (2.0 * L) * (conjg(q0) * s0 + q0 * conjg(s0));
        f[1] = 2.0 * f0 * t.x;
        const double2 u = q0 + rk * s1 - s0;
        f[2] = 2.0 * f0 * (L * abs2(u) + 3.0 * abs2(rk * q1) + L * (l - 1) * (l + 2) * abs2(s0));
    } else {
        const double2 t0 = p[0], t1 = p[1], t2 = p[2];
        f[0] = f0 * r2 * L * abs2(t0);
        const double2 t = L * r2 * (conjg(t0) * t2) + (2.0 * rk * L) * (conjg(t0) * t1) + (-(L * L)) * (conjg(t0) * t0);
        f[1] = 2.0 * f0 * t.x;
        f[2] = 2.0 * f0 * (L * abs2(rk * t1 - t0) + L * (l - 1) * (l + 2) * abs2(t0));
    }
}

// Sums over k = role, role + R, ... of E_j[k][i] c_k for ND derivatives and KV vectors.
template <int ND, int KV, int R>
__device__ __forceinline__ void role_sums(const double *__restrict__ E, int64_t NN, int nh, int N, int i, int role,
                                          const double2 *cs, double2 (&s)[KV][4]) {
#pragma unroll 2
    for (int k = role; k < N; k += R) {
        double ev[ND];
#pragma unroll
        for (int j = 0; j < ND; ++j) ev[j] = __ldg(E + j * NN + (int64_t)k * nh + i);
#pragma unroll
        for (int v = 0; v < KV; ++v) {
            const double2 c = cs[v * N + k];
#pragma unroll
            for (int j = 0; j < ND; ++j) {
                s[v][j].x = fma(ev[j], c.x, s[v][j].x);
                s[v][j].y = fma(ev[j], c.y, s[v][j].y);
            }
        }
    }
}

// pts point pairs at a time (a multiple of 32), R threads each.
template <int KV, int R>
__global__ void __launch_bounds__(kDiagThreads) k_flow_integrals(FlowArgs a, int pts) {
    extern __shared__ double2 cs[];      // KV x N coefficients, then the roles' sums
    __shared__ double red[KV][3][kDiagThreads / 32];
    const int b = blockIdx.x, v0 = blockIdx.y * KV, N = a.N, nh = (N + 1) / 2;
    double2 *ps = cs + KV * N;           // [vector][derivative][role][point]
    const int nblk = a.npol + a.ntor;
    const bool tor = b >= a.npol;
    const int l = tor ? a.ltor[b - a.npol] : a.lpol[b];
    for (int v = 0; v < KV; ++v) {
        const double2 *c = a.x + (v0 + v) * a.vstride + (int64_t)b * N * a.cstride;
        for (int k = threadIdx.x; k < N; k += blockDim.x)
            cs[v * N + k] = v0 + v < a.nvec ? c[k * a.cstride] : mk(0.0, 0.0);
    }
    __syncthreads();
    const int64_t NN = (int64_t)N * nh;
    const int pt = threadIdx.x % pts, role = threadIdx.x / pts;
    double sum[KV][3];
#pragma unroll
    for (int v = 0; v < KV; ++v) sum[v][0] = sum[v][1] = sum[v][2] = 0.0;
    for (int i0 = 0; i0 < nh; i0 += pts) {
        const int i = i0 + pt;
        double2 s[KV][4];
#pragma unroll
        for (int v = 0; v < KV; ++v)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[v][j] = mk(0.0, 0.0);
        if (i < nh) {
            if (tor) role_sums<3, KV, R>(a.E, NN, nh, N, i, role, cs, s);
            else role_sums<4, KV, R>(a.E, NN, nh, N, i, role, cs, s);
        }
        __syncthreads();
#pragma unroll
        for (int v = 0; v < KV; ++v)
#pragma unroll
            for (int j = 0; j < 4; ++j) ps[((v * 4 + j) * R + role) * pts + pt] = s[v][j];
        __syncthreads();
        // role 0 takes x, role 1 its mirror image (the middle point of an odd N has none)
        if (role < 2 && i < nh && !(role == 1 && 2 * i + 1 == N)) {
            const double x = a.E[4 * NN + i], w = a.E[4 * NN + nh + i];
            const double rk = 0.5 * (a.rcmb - a.ricb) * ((role ? -x : x) + 1.0) + a.ricb;
#pragma unroll
            for (int v = 0; v < KV; ++v) {
                double2 p[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    double2 e = mk(0.0, 0.0), o = mk(0.0, 0.0);
#pragma unroll
                    for (int q = 0; q < R; q += 2) {
                        e = e + ps[((v * 4 + j) * R + q) * pts + pt];
                        o = o + ps[((v * 4 + j) * R + q + 1) * pts + pt];
                    }
                    p[j] = role ? e - o : e + o;
                    if (role && (j & 1)) p[j] = -p[j];
                }
                double f[3];
                flow_integrands(tor, l, rk, p, f);
#pragma unroll
                for (int q = 0; q < 3; ++q) sum[v][q] += w * f[q];
            }
        }
    }
#pragma unroll
    for (int v = 0; v < KV; ++v)
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const double t = warp_sum_d(sum[v][q]);
            if ((threadIdx.x & 31) == 0) red[v][q][threadIdx.x >> 5] = t;
        }
    __syncthreads();
    if (threadIdx.x < 3 * KV) {
        const int v = threadIdx.x / 3, q = threadIdx.x - 3 * v;
        if (v0 + v < a.nvec) {
            double t = 0.0;
            for (int w = 0; w < 2 * pts / 32; ++w) t += red[v][q][w];   // roles 0 and 1
            const double quad = (3.14159265358979323846 / N) * (a.rcmb - a.ricb) / 2.0;
            a.out[((int64_t)(v0 + v) * nblk + b) * 3 + q] = quad * t;
        }
    }
}

template <int KV, int R>
int launch_flow(const FlowArgs &a, int device, int pts) {
    const size_t smem = ((size_t)KV * a.N + (size_t)KV * 4 * R * pts) * sizeof(double2);
    KORE_TRY(kore_allow_max_dyn_smem(k_flow_integrals<KV, R>, device));
    k_flow_integrals<KV, R><<<dim3(a.npol + a.ntor, kore_div_up(a.nvec, KV)), R * pts, smem>>>(a, pts);
    return KORE_OK;
}

int flow_diagnostics(int device, int N, double ricb, int npol, const int32_t *lpol, int ntor, const int32_t *ltor,
                     const double *x, int nvec, double *out, bool cols) {
    if (N < 2 || N > 3000 || !(ricb > 0.0 && ricb < 1.0) || npol < 0 || ntor < 0 || npol + ntor == 0 ||
        (npol && !lpol) || (ntor && !ltor) || !x || nvec <= 0 || !out)
        return KORE_EINVAL;
    for (int b = 0; b < npol; ++b) if (lpol[b] < 1) return KORE_EINVAL;
    for (int b = 0; b < ntor; ++b) if (ltor[b] < 1) return KORE_EINVAL;
    int prev = -1;
    cudaGetDevice(&prev);
    if (prev != device) KORE_CUDA_TRY(cudaSetDevice(device));
    const int nblk = npol + ntor;
    const size_t xbytes = (size_t)nvec * nblk * N * sizeof(double2);
    const size_t obytes = (size_t)nvec * nblk * 3 * sizeof(double);
    double *dE = nullptr, *dout = nullptr;
    double2 *dx = nullptr;
    int *dl = nullptr;
    int rc = KORE_OK;
    auto ck = [&](cudaError_t e) {
        if (e != cudaSuccess && rc == KORE_OK) rc = (e == cudaErrorMemoryAllocation) ? KORE_ENOMEM : KORE_ECUDA;
    };
    const int nh = (N + 1) / 2;
    ck(cudaMalloc(&dE, ((size_t)4 * N * nh + 2 * nh) * sizeof(double)));
    ck(cudaMalloc(&dx, xbytes));
    ck(cudaMalloc(&dout, obytes));
    ck(cudaMalloc(&dl, (size_t)nblk * sizeof(int)));
    if (rc == KORE_OK) {
        std::vector<int> ls(lpol, lpol + npol);
        ls.insert(ls.end(), ltor, ltor + ntor);
        ck(cudaMemcpy(dl, ls.data(), ls.size() * sizeof(int), cudaMemcpyHostToDevice));
        ck(cudaMemcpy(dx, x, xbytes, cudaMemcpyHostToDevice));
        k_cheb_eval<<<kore_div_up(nh, 32), 32>>>(N, ricb, 1.0, dE);
        FlowArgs a{N, npol, ntor, nvec, ricb, 1.0, dl, dl + npol, dx, cols ? 1 : (int64_t)nblk * N, cols ? nvec : 1, dE,
                   dout};
        int nsm = 0;
        ck(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device));
        // Many blocks: two vectors share a CTA's reads of E.  Few: the chain of products of
        // one thread is the time, so eight threads share a pair of points.  Whole calls, two
        // vectors and two threads against one and eight: 60 blocks of N = 96, 8 vectors, 380
        // and 417 us; 100 of N = 200, 4 vectors, 608 and 606 us; 300 of N = 240, one vector,
        // 530 and 435 us; 600 of N = 400, one vector, 1,828 and 1,248 us.
        const bool many = nvec > 1 && (int64_t)nblk * nvec >= 2LL * nsm;
        const int pts = std::min(many ? 256 : 64, (nh + 31) / 32 * 32);
        if (rc == KORE_OK) rc = many ? launch_flow<2, 2>(a, device, pts) : launch_flow<1, 8>(a, device, pts);
        KORE_LAUNCHED(2);
        ck(cudaGetLastError());
        ck(cudaMemcpy(out, dout, obytes, cudaMemcpyDeviceToHost));
    }
    cudaFree(dE); cudaFree(dx); cudaFree(dout); cudaFree(dl);
    if (prev >= 0 && prev != device) cudaSetDevice(prev);
    return rc;
}

}  // namespace

extern "C" int kore_flow_diagnostics(int device, int N, double ricb, int npol, const int32_t *lpol, int ntor,
                                     const int32_t *ltor, const double *x, int nvec, double *out) {
    return flow_diagnostics(device, N, ricb, npol, lpol, ntor, ltor, x, nvec, out, false);
}

extern "C" int kore_flow_diagnostics_cols(int device, int N, double ricb, int npol, const int32_t *lpol, int ntor,
                                          const int32_t *ltor, const double *x, int nvec, double *out) {
    return flow_diagnostics(device, N, ricb, npol, lpol, ntor, ltor, x, nvec, out, true);
}
