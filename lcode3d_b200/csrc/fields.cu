// Spectral field solvers: right-hand sides, eigenvalues, the choice of the
// transforms' form (float64 FFT: fields_fft64.cu, float64 dense:
// fields_dense.cu, float32 FFT: fields_fft.cu, split tensor-core GEMMs:
// fields_mixed.cu) and the step finalize.
//
// Reference: lcode.py:124-184 (dst2d, dirichlet_matrix, calculate_Ez),
// 187-290 (mix2d, mixed_matrix, dx_dy, calculate_Ex_Ey_Bx_By), 293-364
// (dct2d, neumann_matrix, calculate_Bz).
//
// The reference builds DST-I / DCT-I out of padded real FFTs. Those
// transforms are linear maps with fixed matrices, so every solve is
//     F = L (Lambda o (L X R)) R
// with X the right-hand side, L / R the transform along axis 0 / axis 1 and
// Lambda the eigenvalue matrix (normalisation folded in):
//     S2[k][n] = 2 sin(pi (k+1)(n+1) / (N-1))            (DST-I, M = N-2)
//     C[k][n]  = c_n cos(pi k n / (N-1)), c_0 = c_{N-1} = 1, else 2   (DCT-I)
//   Ey, Bx: X = rhs[1:-1, :]      L = S2, R = C^T, Lambda = mixed_matrix
//   Ex, By: X = rhs[:, 1:-1]      L = C,  R = S2,  Lambda = mixed_matrix^T
//           (the reference solves them transposed, lcode.py:287-288)
//   Ez:     X = rhs_inner         L = S2, R = S2,  Lambda = dirichlet_matrix
//   Bz:     X = rhs               L = C,  R = C^T, Lambda = neumann_matrix
//           (dct2d is minus the DCT-I; the two signs cancel)
// All six fields of a solve run in each launch.

#include <cmath>
#include <cstring>
#include <vector>

#include "lc3d_internal.cuh"

#ifndef LC3D_FFT32_STREAMS
#define LC3D_FFT32_STREAMS 3   // float32 FFT passes of a solve on 1, 2 or 3 streams
#endif
#ifndef LC3D_FIN_PER_GROUP
#define LC3D_FIN_PER_GROUP 1
#endif

namespace {

// ---------------------------------------------------------------------------
// Right-hand sides, lcode.py:166-168, 234-268, 339-343.
// ---------------------------------------------------------------------------
struct RhsArgs {
    SolveInputs in;
    double st, h, dxi;
    double inv_h2, inv_dxi;   // 1 / (2 h), 1 / dxi
    double* out[6];       // Ex Ey Ez Bx By Bz right-hand sides (N x N, may be NULL)
    int N;
};

__device__ __forceinline__ double avg_in(const double* a, const double* a_prev, size_t k) {
    return a_prev ? (a[k] + a_prev[k]) / 2 : a[k];
}

// x / d from the reciprocal: q0 = x (1/d) is within an ulp of the quotient and
// one correction with the exact residual fma(-q0, d, x) rounds it (the
// float64 divisions of the reference, without the division sequence).
__device__ __forceinline__ double div_by(double x, double d, double inv_d) {
    const double q0 = x * inv_d;
    return fma(fma(-q0, d, x), inv_d, q0);
}

// One grid row per grid line i (blockIdx.y), 128 cells of it per CTA: the
// cell's coordinates come without an integer division.
constexpr int RHS_THREADS = 128;

__global__ void __launch_bounds__(RHS_THREADS) rhs_kernel(const __grid_constant__ RhsArgs a) {
    pdl_wait();
    const int N = a.N;
    const int i = blockIdx.y, j = blockIdx.x * RHS_THREADS + threadIdx.x;
    if (j >= N) return;
    const int k = i * N + j;
    const bool interior = i >= 1 && i <= N - 2 && j >= 1 && j <= N - 2;
    const SolveInputs& in = a.in;
    const double h2 = a.h * 2;
    // every result first, then the stores: the stores could alias the
    // inputs for the compiler, so loads after a store would wait for it
    double o[6] = {};
    if (a.out[0]) {   // the four transverse fields
        double dro_dx = 0, dro_dy = 0, djz_dx = 0, djz_dy = 0;
        if (interior) {
            // (ro_in + beam_ro) and (jz_in + beam_ro) at the four neighbours
            const size_t kp = k + N, km = k - N, lp = k + 1, lm = k - 1;
            dro_dx = div_by((avg_in(in.ro, in.ro_prev, kp) + in.beam[kp]) -
                            (avg_in(in.ro, in.ro_prev, km) + in.beam[km]), h2, a.inv_h2);
            dro_dy = div_by((avg_in(in.ro, in.ro_prev, lp) + in.beam[lp]) -
                            (avg_in(in.ro, in.ro_prev, lm) + in.beam[lm]), h2, a.inv_h2);
            djz_dx = div_by((avg_in(in.jz, in.jz_prev, kp) + in.beam[kp]) -
                            (avg_in(in.jz, in.jz_prev, km) + in.beam[km]), h2, a.inv_h2);
            djz_dy = div_by((avg_in(in.jz, in.jz_prev, lp) + in.beam[lp]) -
                            (avg_in(in.jz, in.jz_prev, lm) + in.beam[lm]), h2, a.inv_h2);
        }
        const double djx_dxi = div_by(in.jx_prev[k] - in.jx[k], a.dxi, a.inv_dxi);
        const double djy_dxi = div_by(in.jy_prev[k] - in.jy[k], a.dxi, a.inv_dxi);
        const double st = a.st;
        o[0] = -((dro_dx - djx_dxi) - in.Ex_sub[k] * st);
        o[1] = -((dro_dy - djy_dxi) - in.Ey_sub[k] * st);
        o[3] = +((djz_dy - djy_dxi) + in.Bx_sub[k] * st);
        o[4] = -((djz_dx - djx_dxi) - in.By_sub[k] * st);
    }
    if (a.out[2] || a.out[5]) {
        double ez = 0, bz = 0;
        if (interior) {
            const double djx_dx = in.jx[k + N] - in.jx[k - N];
            const double djy_dy = in.jy[k + 1] - in.jy[k - 1];
            const double djx_dy = in.jx[k + 1] - in.jx[k - 1];
            const double djy_dx = in.jy[k + N] - in.jy[k - N];
            ez = -div_by(djx_dx + djy_dy, h2, a.inv_h2);
            bz = -div_by(djx_dy - djy_dx, h2, a.inv_h2);
        }
        o[2] = ez;
        o[5] = bz;
    }
#pragma unroll
    for (int f = 0; f < 6; ++f)
        if (a.out[f]) a.out[f][k] = o[f];
}

// ---------------------------------------------------------------------------
// The same right-hand sides straight from a deposition's accumulators, in a
// step: the densities themselves are wanted nowhere else, so neither they nor
// a finalize pass exist there. A CTA converts the accumulators of 32 x 4 cells
// and one more on each side, averages and adds the beam once per cell, and
// keeps the four quantities in shared memory for the differences. It also
// clears its cells of the other accumulators, those of the next deposition.
// Bound by latency and the L2: 641^2 69 MB read, 46 MB written in 19.5 us
// (32 x 8 cells on 256 threads 21.2, 32 x 16 on 512 21.6); a finalize pass and
// rhs_kernel take 11.5 + 13.2.
// ---------------------------------------------------------------------------
constexpr int RA_X = 32, RA_Y = 4, RA_W = RA_X + 2, RA_CELLS = RA_W * (RA_Y + 2), RA_THREADS = RA_X * RA_Y;

__global__ void __launch_bounds__(RA_THREADS, 7) rhs_acc_kernel(const __grid_constant__ RhsArgs a, size_t plane) {
    __shared__ double s_ro[RA_CELLS], s_jz[RA_CELLS], s_jx[RA_CELLS], s_jy[RA_CELLS];
    const int N = a.N, t = threadIdx.x;
    const int i0 = blockIdx.y * RA_Y - 1, j0 = blockIdx.x * RA_X - 1;
    const SolveInputs& in = a.in;
    constexpr int PER = (RA_CELLS + RA_THREADS - 1) / RA_THREADS;
    const int i = i0 + 1 + t / RA_X, j = j0 + 1 + t % RA_X;   // this thread's cell
    const bool live = i < N && j < N;
    const int k = i * N + j;
    pdl_wait();
    // every load first: the accumulators and what is added to them, then the
    // cell's own terms
    unsigned long long w[PER][DEP_WORDS_PER_CELL];
    double ri[PER], rp[PER], zp[PER], bm[PER];
    bool ok[PER];
#pragma unroll
    for (int u = 0; u < PER; ++u) {
        const int c = t + u * RA_THREADS, ci = i0 + c / RA_W, cj = j0 + c % RA_W;
        ok[u] = c < RA_CELLS && ci >= 0 && ci < N && cj >= 0 && cj < N;
        if (!ok[u]) continue;
        const int g = ci * N + cj;
#pragma unroll
        for (int q = 0; q < DEP_WORDS_PER_CELL; ++q) w[u][q] = __ldcg(in.acc + q * plane + g);
        ri[u] = __ldg(in.ro_initial + g);
        rp[u] = in.ro_prev ? __ldg(in.ro_prev + g) : 0.0;
        zp[u] = in.jz_prev ? __ldg(in.jz_prev + g) : 0.0;
        bm[u] = __ldg(in.beam + g);
    }
    double xp = 0, yp = 0, sub[4] = {};
    if (live) {
        xp = __ldg(in.jx_prev + k);
        yp = __ldg(in.jy_prev + k);
        sub[0] = __ldg(in.Ex_sub + k);
        sub[1] = __ldg(in.Ey_sub + k);
        sub[2] = __ldg(in.Bx_sub + k);
        sub[3] = __ldg(in.By_sub + k);
    }
#pragma unroll
    for (int u = 0; u < PER; ++u) {
        if (!ok[u]) continue;
        const int c = t + u * RA_THREADS;
        double v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = fx_value((long long)w[u][2 * q], (long long)w[u][2 * q + 1]);
        v[0] += ri[u];
        s_ro[c] = (in.ro_prev ? (v[0] + rp[u]) / 2 : v[0]) + bm[u];
        s_jz[c] = (in.jz_prev ? (v[3] + zp[u]) / 2 : v[3]) + bm[u];
        s_jx[c] = v[1];
        s_jy[c] = v[2];
    }
    __syncthreads();
    if (!live) return;
    const int c = (t / RA_X + 1) * RA_W + t % RA_X + 1;
    const double h2 = a.h * 2, st = a.st;
    double o[6];
    double dro_dx = 0, dro_dy = 0, djz_dx = 0, djz_dy = 0;
    o[2] = o[5] = 0;
    if (i >= 1 && i <= N - 2 && j >= 1 && j <= N - 2) {
        dro_dx = div_by(s_ro[c + RA_W] - s_ro[c - RA_W], h2, a.inv_h2);
        dro_dy = div_by(s_ro[c + 1] - s_ro[c - 1], h2, a.inv_h2);
        djz_dx = div_by(s_jz[c + RA_W] - s_jz[c - RA_W], h2, a.inv_h2);
        djz_dy = div_by(s_jz[c + 1] - s_jz[c - 1], h2, a.inv_h2);
        const double djx_dx = s_jx[c + RA_W] - s_jx[c - RA_W];
        const double djy_dy = s_jy[c + 1] - s_jy[c - 1];
        const double djx_dy = s_jx[c + 1] - s_jx[c - 1];
        const double djy_dx = s_jy[c + RA_W] - s_jy[c - RA_W];
        o[2] = -div_by(djx_dx + djy_dy, h2, a.inv_h2);
        o[5] = -div_by(djx_dy - djy_dx, h2, a.inv_h2);
    }
    const double djx_dxi = div_by(xp - s_jx[c], a.dxi, a.inv_dxi);
    const double djy_dxi = div_by(yp - s_jy[c], a.dxi, a.inv_dxi);
    o[0] = -((dro_dx - djx_dxi) - sub[0] * st);
    o[1] = -((dro_dy - djy_dxi) - sub[1] * st);
    o[3] = +((djz_dy - djy_dxi) + sub[2] * st);
    o[4] = -((djz_dx - djx_dxi) - sub[3] * st);
#pragma unroll
    for (int f = 0; f < 6; ++f) a.out[f][k] = o[f];
#pragma unroll
    for (int q = 0; q < DEP_WORDS_PER_CELL; ++q) __stcg(in.acc_clear + q * plane + k, 0ull);
}

// ---------------------------------------------------------------------------
// Deterministic mean (fixed summation tree) and the step finalisation.
// ---------------------------------------------------------------------------
constexpr int RED_THREADS = 256;

__device__ __forceinline__ double block_sum_fixed(double v, double* sh) {
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int s = RED_THREADS / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
        __syncthreads();
    }
    return sh[0];
}

__global__ void __launch_bounds__(RED_THREADS) partial_sum_kernel(const double* __restrict__ a, int n,
                                                                  double* __restrict__ partial) {
    pdl_wait();
    __shared__ double sh[RED_THREADS];
    double v = 0;
    for (int k = blockIdx.x * RED_THREADS + threadIdx.x; k < n; k += gridDim.x * RED_THREADS) v += a[k];
    double s = block_sum_fixed(v, sh);
    if (threadIdx.x == 0) partial[blockIdx.x] = s;
}

__device__ double mean_from_partials(const double* partial, int nblocks, double inv_n, double* sh) {
    double v = 0;
    for (int k = threadIdx.x; k < nblocks; k += RED_THREADS) v += partial[k];
    return block_sum_fixed(v, sh) * inv_n;
}

struct FinalizeArgs {
    const double* raw[6];
    const double* prev[6];
    double* out[6];
    double* avg[6];
    const double* partial;
    int nblocks, n, variant_A, has_bz;
    int vec;                          // set by the launcher: every array 16-byte aligned, two cells per thread
    double inv_n;
};

// Field f of one cell: the mean-free Bz, Variant A's 2 F - F_prev, and the
// half-step average (lcode.py:876-881, 906-911).
__device__ __forceinline__ double2 finalize_value(const FinalizeArgs& a, int f, double raw, double prev, double mean) {
    double v = raw;
    if (f == 5) v -= mean;
    if (a.variant_A && f != 2 && f != 5) v = 2 * v - prev;
    return make_double2(v, (v + prev) / 2);
}

__global__ void __launch_bounds__(RED_THREADS) finalize_step_kernel(const __grid_constant__ FinalizeArgs a) {
    pdl_wait();
    __shared__ double sh[RED_THREADS];
    int k = blockIdx.x * RED_THREADS + threadIdx.x;
    if (a.vec) {
        // two cells per thread: all twelve 16-byte loads issued before the
        // stores, and before the Bz mean's reduction (which they overlap)
        k *= 2;
        const bool pair = k + 1 < a.n;
        double2 r[6], p[6];
        if (pair) {
#pragma unroll
            for (int f = 0; f < 6; ++f)
                if (a.raw[f]) {
                    r[f] = __ldcg(reinterpret_cast<const double2*>(a.raw[f] + k));
                    p[f] = __ldcg(reinterpret_cast<const double2*>(a.prev[f] + k));
                }
        }
        // every thread of the CTA takes part in the reduction's barriers
        const double mean = a.has_bz ? mean_from_partials(a.partial, a.nblocks, a.inv_n, sh) : 0.0;
        if (k >= a.n) return;
        if (pair) {
#pragma unroll
            for (int f = 0; f < 6; ++f) {
                if (!a.raw[f]) continue;
                const double2 v0 = finalize_value(a, f, r[f].x, p[f].x, mean);
                const double2 v1 = finalize_value(a, f, r[f].y, p[f].y, mean);
                if (a.out[f]) *reinterpret_cast<double2*>(a.out[f] + k) = make_double2(v0.x, v1.x);
                *reinterpret_cast<double2*>(a.avg[f] + k) = make_double2(v0.y, v1.y);
            }
            return;
        }
        // an odd cell count leaves the last cell to one thread
#pragma unroll
        for (int f = 0; f < 6; ++f) {
            if (!a.raw[f]) continue;
            const double2 v = finalize_value(a, f, a.raw[f][k], a.prev[f][k], mean);
            if (a.out[f]) a.out[f][k] = v.x;
            a.avg[f][k] = v.y;
        }
        return;
    }
    const double mean = a.has_bz ? mean_from_partials(a.partial, a.nblocks, a.inv_n, sh) : 0.0;
    if (k >= a.n) return;
#pragma unroll
    for (int f = 0; f < 6; ++f) {
        if (!a.raw[f]) continue;
        const double2 v = finalize_value(a, f, a.raw[f][k], a.prev[f][k], mean);
        if (a.out[f]) a.out[f][k] = v.x;
        a.avg[f][k] = v.y;
    }
}

__global__ void __launch_bounds__(RED_THREADS) subtract_mean_kernel(double* a, int n, const double* partial,
                                                                    int nblocks, double inv_n) {
    pdl_wait();
    __shared__ double sh[RED_THREADS];
    const double mean = mean_from_partials(partial, nblocks, inv_n, sh);
    const int k = blockIdx.x * RED_THREADS + threadIdx.x;
    if (k < n) a[k] -= mean;
}

// ---------------------------------------------------------------------------
// Host: eigenvalue matrices.
// ---------------------------------------------------------------------------

// lam[k] = 4 / h**2 * sin(k pi / (2 (N - 1)))**2 as lcode.py:152-154 writes it
double lam(int k, int N, double h) {
    double s = std::sin(k * M_PI / (2.0 * (N - 1)));
    return 4 / (h * h) * (s * s);
}

int upload(double** dst, const std::vector<double>& v) {
    LC3D_CUDA_TRY(cudaMalloc(dst, v.size() * sizeof(double)));
    LC3D_CUDA_TRY(cudaMemcpy(*dst, v.data(), v.size() * sizeof(double), cudaMemcpyHostToDevice));
    return LC3D_OK;
}

// float copy of an eigenvalue matrix (float32-transform precision)
int upload32(float** dst, const std::vector<double>& v) {
    std::vector<float> f(v.begin(), v.end());
    LC3D_CUDA_TRY(cudaMalloc(dst, f.size() * sizeof(float)));
    LC3D_CUDA_TRY(cudaMemcpy(*dst, f.data(), f.size() * sizeof(float), cudaMemcpyHostToDevice));
    return LC3D_OK;
}

}  // namespace

int fields_init(lc3d_ctx* c) {
    const int N = c->N, M = c->M;
    const double h = c->p.grid_step_size;
    const double norm = 1.0 / ((2.0 * (N - 1)) * (2.0 * (N - 1)));
    const double trick = c->p.field_solver_subtraction_trick != 0 ? 1.0 : 0.0;
    std::vector<double> ld((size_t)M * M), lm((size_t)M * N), lmT((size_t)N * M), ln((size_t)N * N);
    std::vector<double> lamk(N);
    for (int k = 0; k < N; ++k) lamk[k] = lam(k, N, h);
    for (int i = 0; i < M; ++i)
        for (int j = 0; j < M; ++j) ld[(size_t)i * M + j] = (1 / (lamk[i + 1] + lamk[j + 1])) * norm;
    for (int i = 0; i < M; ++i)
        for (int j = 0; j < N; ++j) {
            const double v = (1 / (lamk[i + 1] + lamk[j] + trick)) * norm;
            lm[(size_t)i * N + j] = v;
            lmT[(size_t)j * M + i] = v;
        }
    for (int i = 0; i < N; ++i)
        for (int j = 0; j < N; ++j)
            ln[(size_t)i * N + j] = (i == 0 && j == 0) ? 0.0 : (1 / (lamk[i] + lamk[j])) * norm;
    if (c->p.precision != LC3D_PREC_FFT32) {
        LC3D_TRY(upload(&c->lam_dir, ld));
        LC3D_TRY(upload(&c->lam_mix, lm));
        LC3D_TRY(upload(&c->lam_mixT, lmT));
        LC3D_TRY(upload(&c->lam_neu, ln));
    } else {
        LC3D_TRY(upload32(&c->lam32_dir, ld));
        LC3D_TRY(upload32(&c->lam32_mix, lm));
        LC3D_TRY(upload32(&c->lam32_mixT, lmT));
        LC3D_TRY(upload32(&c->lam32_neu, ln));
    }
    const size_t plane = (size_t)N * N * sizeof(double);
    const size_t tplane = (size_t)N * fft64_pitch(N) * sizeof(double);   // the transform intermediates
    for (int f = 0; f < 6; ++f) {
        LC3D_CUDA_TRY(cudaMalloc(&c->rhs[f], plane));
        LC3D_CUDA_TRY(cudaMalloc(&c->t1[f], tplane));
        LC3D_CUDA_TRY(cudaMalloc(&c->t2[f], tplane));
        LC3D_CUDA_TRY(cudaMemset(c->t1[f], 0, tplane));
        LC3D_CUDA_TRY(cudaMemset(c->t2[f], 0, tplane));
        LC3D_CUDA_TRY(cudaMemset(c->rhs[f], 0, plane));
        if (c->use_fft && c->p.precision == LC3D_PREC_FP64) continue;   // these solves write the fields themselves
        LC3D_CUDA_TRY(cudaMalloc(&c->raw[f], plane));
        LC3D_CUDA_TRY(cudaMemset(c->raw[f], 0, plane));
    }
    c->red_blocks = 160;
    // room for the partial-sum kernel's blocks and for the FFT pass's per-CTA sums
    LC3D_CUDA_TRY(cudaMalloc(&c->red, 4096 * sizeof(double)));
    return LC3D_OK;
}

void fields_drop_lam(lc3d_ctx* c) {
    double** ps[] = {&c->lam_dir, &c->lam_mix, &c->lam_mixT, &c->lam_neu};
    for (double** p : ps) {
        if (*p) cudaFree(*p);
        *p = nullptr;
    }
}

void fields_free(lc3d_ctx* c) {
    fields_drop_lam(c);
    if (c->red) cudaFree(c->red);
    c->red = nullptr;
    float** ps32[] = {&c->lam32_dir, &c->lam32_mix, &c->lam32_mixT, &c->lam32_neu};
    for (float** p : ps32) {
        if (*p) cudaFree(*p);
        *p = nullptr;
    }
    for (int f = 0; f < 6; ++f) {
        double** q[] = {&c->rhs[f], &c->t1[f], &c->t2[f], &c->raw[f]};
        for (double** p : q) {
            if (*p) cudaFree(*p);
            *p = nullptr;
        }
    }
}

namespace {

struct FieldGeom {
    int rows, cols;
    size_t off;            // offset of X / output inside an N x N plane
    const double* Lam;
    int ldLam;
    int type0, type1;      // axis-0 / axis-1 transform: 0 DCT-I, 1 DST-I
};

FieldGeom geom(const lc3d_ctx* c, int f) {
    const int N = c->N, M = c->M;
    FieldGeom g{};
    switch (f) {
        case 0: case 4:   // Ex, By: solved transposed
            g = {N, M, 1, c->lam_mixT, M, 0, 1};
            break;
        case 1: case 3:   // Ey, Bx
            g = {M, N, (size_t)N, c->lam_mix, N, 1, 0};
            break;
        case 2:           // Ez
            g = {M, M, (size_t)N + 1, c->lam_dir, M, 1, 1};
            break;
        default:          // Bz
            g = {N, N, 0, c->lam_neu, N, 0, 0};
            break;
    }
    return g;
}

// The float copy of field f's eigenvalue matrix (float32-transform precision).
const float* lam32(const lc3d_ctx* c, int f) {
    switch (f) {
        case 0: case 4: return c->lam32_mixT;
        case 1: case 3: return c->lam32_mix;
        case 2: return c->lam32_dir;
        default: return c->lam32_neu;
    }
}

}  // namespace

int solve_fields(lc3d_ctx* c, int which, const SolveInputs& in, const SolveOutputs& o, cudaStream_t s) {
    const int N = c->N;
    const int n = N * N;
    bool on[6] = {false, false, false, false, false, false};
    if (which & LC3D_F_EXEYBXBY) on[0] = on[1] = on[3] = on[4] = true;
    if (which & LC3D_F_EZ) on[2] = true;
    if (which & LC3D_F_BZ) on[5] = true;

    RhsArgs ra{};
    memset(&ra, 0, sizeof(ra));
    ra.in = in;
    ra.st = c->p.field_solver_subtraction_trick;
    ra.h = c->p.grid_step_size;
    ra.dxi = c->p.xi_step_size;
    ra.inv_h2 = 1.0 / (ra.h * 2);
    ra.inv_dxi = 1.0 / ra.dxi;
    ra.N = N;
    for (int f = 0; f < 6; ++f) ra.out[f] = on[f] ? c->rhs[f] : nullptr;
    {
        ProfScope ps(c, LC3D_STAGE_RHS, s);
        if (in.acc)
            LC3D_CUDA_TRY(launch_pdl(rhs_acc_kernel, dim3((N + RA_X - 1) / RA_X, (N + RA_Y - 1) / RA_Y),
                                     dim3(RA_THREADS), 0, s, ra, c->acc_plane));
        else
            LC3D_CUDA_TRY(launch_pdl(rhs_kernel, dim3((N + RHS_THREADS - 1) / RHS_THREADS, N), dim3(RHS_THREADS), 0,
                                     s, ra));
        LC3D_CUDA_TRY(cudaGetLastError());
    }

    if (c->use_fft && c->p.precision == LC3D_PREC_FP64) {
        Fft64Desc d[6]{};
        int cnt = 0;
        for (int f = 0; f < 6; ++f) {
            if (!on[f]) continue;
            const FieldGeom g = geom(c, f);
            Fft64Desc& e = d[cnt++];
            e.rhs = c->rhs[f];
            e.type0 = g.type0;
            e.type1 = g.type1;
            e.t1 = c->t1[f];
            e.t2 = c->t2[f];
            e.out = o.out[f];
            if (o.mode == 1) {
                e.prev = o.prev[f];
                e.avg = o.avg[f];
                e.variant_a = c->p.field_solver_variant_A && f != 2 && f != 5;
            }
            e.sums = f == 5 ? c->red : nullptr;
        }
        return fft64_solve(c, d, cnt, s);
    }

    // destination of the raw solution
    double* dst[6];
    for (int f = 0; f < 6; ++f) {
        dst[f] = nullptr;
        if (!on[f]) continue;
        if (o.mode == 0) {
            dst[f] = o.out[f];
            if (f != 5) LC3D_CUDA_TRY(cudaMemsetAsync(dst[f], 0, (size_t)n * sizeof(double), s));
        } else {
            dst[f] = c->raw[f];
        }
    }
    int bz_partials = 0;   // > 0: the FFT pass left this many Bz partial sums in c->red
    // FFT passes on several streams whose join waits until each group's
    // finalize has run on its own stream (step finalisation only)
    int fin_groups = 0;
    int fin_group_of[6] = {0, 0, 0, 0, 0, 0};
    cudaStream_t fin_stream[3] = {s, s, s};
    if (c->p.precision == LC3D_PREC_MIXED || c->p.precision == LC3D_PREC_TF32) {
        // four split-BF16 tensor-core GEMM stages (fields_mixed.cu)
        for (int stage = 0; stage < 4; ++stage) {
            MixedStageDesc d[6]{};
            int cnt = 0;
            for (int f = 0; f < 6; ++f) {
                if (!on[f]) continue;
                const FieldGeom g = geom(c, f);
                MixedStageDesc& e = d[cnt++];
                memset(&e, 0, sizeof(e));
                e.field = f;
                e.M = g.rows;
                e.N = g.cols;
                e.ld_data = N;
                e.ldo = N;
                const int fixed_L = g.type0 ? 0 : 1, fixed_RT = g.type1 ? 0 : 1;   // 0: S2, 1: C
                switch (stage) {
                    case 0:   // T1^T = (X R)^T
                        e.data = c->rhs[f] + g.off; e.data_rows = g.rows; e.K = g.cols;
                        e.data_is_a = 1; e.fixed = fixed_RT; e.out = c->t1[f]; e.transposed = 1;
                        break;
                    case 1:   // Z = Lambda o (L T1)
                        e.data = c->t1[f]; e.data_rows = g.cols; e.K = g.rows;
                        e.data_is_a = 0; e.fixed = fixed_L; e.out = c->t2[f];
                        e.lam = g.Lam; e.ldl = g.ldLam;
                        break;
                    case 2:   // U^T = (Z R)^T
                        e.data = c->t2[f]; e.data_rows = g.rows; e.K = g.cols;
                        e.data_is_a = 1; e.fixed = fixed_RT; e.out = c->t1[f]; e.transposed = 1;
                        break;
                    default:  // F = L U
                        e.data = c->t1[f]; e.data_rows = g.cols; e.K = g.rows;
                        e.data_is_a = 0; e.fixed = fixed_L; e.out = dst[f] + g.off;
                        break;
                }
            }
            LC3D_TRY(mixed_stage(c, d, cnt, s));
        }
    } else if (c->p.precision == LC3D_PREC_FFT32) {
        // four FFT row passes, each writing its output transposed; the two
        // intermediates (in the t1 / t2 planes) are float32
        static const int types[4] = {FFT_F64_F32, FFT_F32, FFT_F32, FFT_F32_F64};
        // The fields' passes on several streams (forked after the right-hand
        // sides, joined before the finalize): with two, the E fields on the
        // solve's stream and the B fields on a second; with three, Ex Ey /
        // Bx By / Ez Bz. The groups' passes are independent, so the tail of
        // one group's pass, when only part of the SMs still work, is filled
        // by the other groups' row groups. Measured at 641^2: 2109 -> 2145
        // xi-steps/s with two streams, 2176 with three. The per-launch
        // timing pass keeps one stream, and so do the steps of a batch graph
        // (its branches overlap the simulations already).
        const int nstreams = (c->prof_on || c->one_stream) ? 1 : LC3D_FFT32_STREAMS;
        auto group_of = [&](int f) {
            if (nstreams == 3) return f == 2 || f == 5 ? 2 : (f < 2 ? 0 : 1);
            if (nstreams == 2) return f < 3 ? 0 : 1;
            return 0;
        };
        bool used[3] = {false, false, false};
        for (int f = 0; f < 6; ++f)
            if (on[f]) used[group_of(f)] = true;
        if (nstreams > 1) {
            LC3D_CUDA_TRY(cudaEventRecord(c->ev_fork, s));
            for (int q = 1; q < nstreams; ++q)
                if (used[q]) LC3D_CUDA_TRY(cudaStreamWaitEvent(c->fft_stream[q - 1], c->ev_fork, 0));
        }
        for (int stage = 0; stage < 4; ++stage) {
            FftRowsDesc d[6]{};
            int cnt = 0;
            for (int f = 0; f < 6; ++f) {
                if (!on[f]) continue;
                const FieldGeom g = geom(c, f);
                FftRowsDesc& e = d[cnt++];
                memset(&e, 0, sizeof(e));
                e.ld_in = N;
                e.ld_out = N;
                switch (stage) {
                    case 0: e.in = c->rhs[f] + g.off; e.rows = g.rows; e.type = g.type1; e.out = c->t1[f]; break;
                    case 1: e.in = c->t1[f]; e.rows = g.cols; e.type = g.type0; e.out = c->t2[f];
                            e.lam = lam32(c, f);
                            e.ld_lam = g.ldLam; break;   // Lambda o Z as Z is written
                    case 2: e.in = c->t2[f]; e.rows = g.rows; e.type = g.type1; e.out = c->t1[f]; break;
                    default: e.in = c->t1[f]; e.rows = g.cols; e.type = g.type0; e.out = dst[f] + g.off;
                             if (f == 5) {   // Bz: the mean's partial sums come with the last pass
                                 e.partial = c->red;
                                 bz_partials = (g.cols + fft_cta_rows() - 1) / fft_cta_rows();
                             }
                             break;
                }
            }
            if (nstreams > 1) {   // each group of fields on its stream
                for (int q = 0; q < nstreams; ++q) {
                    if (!used[q]) continue;
                    FftRowsDesc dq[6];
                    int nq = 0, k = 0;
                    for (int f = 0; f < 6; ++f) {
                        if (!on[f]) continue;
                        if (group_of(f) == q) dq[nq++] = d[k];
                        ++k;
                    }
                    LC3D_TRY(fft_rows(c, dq, nq, types[stage], q ? c->fft_stream[q - 1] : s));
                }
            } else {
                LC3D_TRY(fft_rows(c, d, cnt, types[stage], s));
            }
        }
        if (LC3D_FIN_PER_GROUP && o.mode == 1 && nstreams > 1) {   // each group finalised on its own stream, then joined
            fin_groups = nstreams;
            for (int f = 0; f < 6; ++f) fin_group_of[f] = group_of(f);
            for (int q = 1; q < nstreams; ++q) fin_stream[q] = used[q] ? c->fft_stream[q - 1] : s;
        } else {
            for (int q = 1; q < nstreams; ++q) {
                if (!used[q]) continue;
                LC3D_CUDA_TRY(cudaEventRecord(c->ev_join[q - 1], c->fft_stream[q - 1]));
                LC3D_CUDA_TRY(cudaStreamWaitEvent(s, c->ev_join[q - 1], 0));
            }
        }
    } else {
        DenseDesc d[6]{};
        int cnt = 0;
        for (int f = 0; f < 6; ++f) {
            if (!on[f]) continue;
            const FieldGeom g = geom(c, f);
            d[cnt++] = {c->rhs[f] + g.off, g.type0, g.type1, c->t1[f], c->t2[f], dst[f] + g.off};
        }
        LC3D_TRY(dense_solve(c, d, cnt, s));
    }
    const double inv_n = 1.0 / n;
    if (on[5] && !bz_partials) {
        ProfScope ps(c, LC3D_STAGE_FIELD_FIN, s);
        LC3D_CUDA_TRY(launch_pdl(partial_sum_kernel, dim3(c->red_blocks), dim3(RED_THREADS), 0, s,
                                 static_cast<const double*>(dst[5]), n, c->red));
        LC3D_CUDA_TRY(cudaGetLastError());
    }
    const int nred = bz_partials ? bz_partials : c->red_blocks;
    if (o.mode == 0) {
        if (on[5]) {
            ProfScope ps(c, LC3D_STAGE_FIELD_FIN, s);
            LC3D_CUDA_TRY(launch_pdl(subtract_mean_kernel, dim3((n + RED_THREADS - 1) / RED_THREADS),
                                     dim3(RED_THREADS), 0, s, dst[5], n, static_cast<const double*>(c->red),
                                     nred, inv_n));
            LC3D_CUDA_TRY(cudaGetLastError());
        }
        return LC3D_OK;
    }
    // one finalize over all fields, or one per group of fields on that
    // group's stream (the groups' FFT passes ran on several streams)
    for (int q = 0; q < (fin_groups ? fin_groups : 1); ++q) {
        FinalizeArgs fa{};
        memset(&fa, 0, sizeof(fa));
        for (int f = 0; f < 6; ++f) {
            if (!on[f] || (fin_groups && fin_group_of[f] != q)) continue;
            fa.raw[f] = c->raw[f];
            fa.prev[f] = o.prev[f];
            fa.out[f] = o.out[f];
            fa.avg[f] = o.avg[f];
        }
        bool any = false;
        for (int f = 0; f < 6; ++f) any = any || fa.raw[f];
        if (!any) continue;
        fa.partial = c->red;
        fa.nblocks = nred;
        fa.n = n;
        fa.variant_A = c->p.field_solver_variant_A;
        fa.has_bz = fa.raw[5] != nullptr;
        fa.inv_n = inv_n;
        uintptr_t al = 0;
        for (int f = 0; f < 6; ++f)
            al |= reinterpret_cast<uintptr_t>(fa.raw[f]) | reinterpret_cast<uintptr_t>(fa.prev[f]) |
                  reinterpret_cast<uintptr_t>(fa.out[f]) | reinterpret_cast<uintptr_t>(fa.avg[f]);
        fa.vec = (al & 15) == 0;
        const int threads = fa.vec ? (n + 1) / 2 : n;
        cudaStream_t sq = fin_groups ? fin_stream[q] : s;
        ProfScope ps(c, LC3D_STAGE_FIELD_FIN, sq);
        LC3D_CUDA_TRY(launch_pdl(finalize_step_kernel, dim3((threads + RED_THREADS - 1) / RED_THREADS),
                                 dim3(RED_THREADS), 0, sq, fa));
        LC3D_CUDA_TRY(cudaGetLastError());
    }
    for (int q = 1; q < fin_groups; ++q) {
        if (fin_stream[q] == s) continue;
        LC3D_CUDA_TRY(cudaEventRecord(c->ev_join[q - 1], fin_stream[q]));
        LC3D_CUDA_TRY(cudaStreamWaitEvent(s, c->ev_join[q - 1], 0));
    }
    return LC3D_OK;
}
