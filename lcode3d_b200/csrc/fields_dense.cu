// Spectral field solves in dense-transform (GEMM) form, float64: grids whose
// 2 (N - 1) has other factors than 2, 3 and 5, and lc3d_fp64_transform =
// 'dense'.
//
// A solve is F = L (Lambda o (L X R)) R with the DST-I / DCT-I matrices of
// fields.cu. Rows of T = S2 or C are even or odd about their centre c,
//     T[k][m - n] = (-1)^k T[k][n],   m the last index,
// so along each axis the even outputs see only x[n] + x[m - n] and the odd
// ones x[n] - x[m - n]: two transforms of half the size, half the products.
// A solve folds X once along both axes (even part first, then odd, in rows
// and in columns), keeps the spectrum sorted by parity (Lambda to match) and
// unfolds once at the end:
//     fold, t1 = X R, t2 = Lambda o (L t1), t1 = t2 R', t2 = L' t1, unfold
// with L, R block diagonal in the parity: 12 GEMMs (6 fields, 2 parities) per
// launch. (' : the matrices of the way back, F[n] = sum_k T[n][k] G[k].)

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "lc3d_internal.cuh"

namespace {

// ---------------------------------------------------------------------------
// Fold and unfold
// ---------------------------------------------------------------------------
struct FoldArgs {
    const double* in[6];
    double* out[6];
    int ld_in, ld_out;
    int rows[6], cols[6];
};

// A folded row: the even part, then the odd part from the next 128-byte line
// on. Every operand of the GEMMs (folded planes, their odd parts, the half
// matrices) has its rows on whole lines, so that copies of 16 bytes apply and
// a k-step of 16 touches one line per row.
__host__ __device__ constexpr int odd_at(int n) { return (n / 2 + 16) & ~15; }          // n odd
__host__ __device__ constexpr int folded_width(int n) { return odd_at(n) + n / 2; }

// One thread per (a, b), a <= (rows - 1) / 2, b <= (cols - 1) / 2 (sizes are
// odd): the four cells it mirrors to, and the four sums and differences. The
// centre is its own mirror and belongs to the even part alone.
__global__ void __launch_bounds__(128) fold_kernel(const __grid_constant__ FoldArgs g) {
    pdl_wait();
    const int f = blockIdx.z, a = blockIdx.y, b = blockIdx.x * blockDim.x + threadIdx.x;
    const int c0 = (g.rows[f] - 1) / 2, c1 = (g.cols[f] - 1) / 2;
    if (a > c0 || b > c1) return;
    const int a2 = g.rows[f] - 1 - a, b2 = g.cols[f] - 1 - b;
    const double* x = g.in[f];
    const double x00 = x[(size_t)a * g.ld_in + b];
    const double x01 = b < c1 ? x[(size_t)a * g.ld_in + b2] : 0.0;
    const double x10 = a < c0 ? x[(size_t)a2 * g.ld_in + b] : 0.0;
    const double x11 = a < c0 && b < c1 ? x[(size_t)a2 * g.ld_in + b2] : 0.0;
    double* o = g.out[f];
    const size_t even = (size_t)a * g.ld_out, odd = (size_t)(c0 + 1 + a) * g.ld_out;
    const int b1 = odd_at(g.cols[f]) + b;
    o[even + b] = (x00 + x01) + (x10 + x11);
    if (b < c1) o[even + b1] = (x00 - x01) + (x10 - x11);
    if (a < c0) o[odd + b] = (x00 + x01) - (x10 + x11);
    if (a < c0 && b < c1) o[odd + b1] = (x00 - x01) - (x10 - x11);
}

// The inverse walk: value and mirrors from the even and odd parts.
__global__ void __launch_bounds__(128) unfold_kernel(const __grid_constant__ FoldArgs g) {
    pdl_wait();
    const int f = blockIdx.z, a = blockIdx.y, b = blockIdx.x * blockDim.x + threadIdx.x;
    const int c0 = (g.rows[f] - 1) / 2, c1 = (g.cols[f] - 1) / 2;
    if (a > c0 || b > c1) return;
    const int a2 = g.rows[f] - 1 - a, b2 = g.cols[f] - 1 - b;
    const double* x = g.in[f];
    const size_t even = (size_t)a * g.ld_in, odd = (size_t)(c0 + 1 + a) * g.ld_in;
    const int b1 = odd_at(g.cols[f]) + b;
    const double ee = x[even + b];
    const double eo = b < c1 ? x[even + b1] : 0.0;
    const double oe = a < c0 ? x[odd + b] : 0.0;
    const double oo = a < c0 && b < c1 ? x[odd + b1] : 0.0;
    double* o = g.out[f];
    o[(size_t)a * g.ld_out + b] = (ee + eo) + (oe + oo);
    if (b < c1) o[(size_t)a * g.ld_out + b2] = (ee - eo) + (oe - oo);
    if (a < c0) o[(size_t)a2 * g.ld_out + b] = (ee + eo) - (oe + oo);
    if (a < c0 && b < c1) o[(size_t)a2 * g.ld_out + b2] = (ee - eo) - (oe - oo);
}

// out[i][j] = lam[k0 of i][k1 of j], both axes sorted by parity, the columns
// as a folded row's (0 between the parts).
__global__ void lam_parity_kernel(const double* __restrict__ lam, int rows, int cols, double* __restrict__ out) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
    const int width = folded_width(cols), j1 = odd_at(cols);
    if (j >= width) return;
    const int e0 = (rows + 1) / 2;
    const int k0 = i < e0 ? 2 * i : 2 * (i - e0) + 1, k1 = j < j1 ? 2 * j : 2 * (j - j1) + 1;
    out[(size_t)i * width + j] = k1 < cols ? lam[(size_t)k0 * cols + k1] : 0.0;
}

// ---------------------------------------------------------------------------
// Batched float64 GEMM, C = A B (optionally C = Lambda o (A B)), row-major,
// on the float64 tensor cores (mma.sync m16n8k8 .f64: float64 products and
// sums throughout). 64 x 32 tiles per 128-thread CTA, a 32 x 16 tile (2 x 2
// MMAs per k8 step) per warp; k-steps of 16 staged by 16-byte cp.async into
// two shared-memory buffers, the next k-step copied while the current one is
// multiplied. Copies go through L1 (.ca): the CTAs of an SM share their
// panels there (an xi step in a graph at 387^2 292 us, past L1 394).
//
// The tile is small because the problems are: at 387^2 a launch has 12 of
// about 387 x 194 x 194, and what is lost is rows and columns past the edges
// and SMs with a tile less than others (a launch at 387^2 28 us; 78 with
// matrices of full size in 128 x 64 tiles of m8n8k4 MMAs). Four warps of
// 32 x 16 a CTA hide more of a k-step's latency than two of 32 x 32: an xi step
// in a graph at 163^2 107 us against 128, 641^2 772 against 911.
// ---------------------------------------------------------------------------
constexpr int MAX_PROBS = 12;

struct GemmProb {
    const double *A, *B, *L;
    double* C;
    int M, N, K, lda, ldb, ldc, ldl;
    int tiles_n, tile_start;
};

struct GemmBatch {
    GemmProb p[MAX_PROBS];
    int count;
};

constexpr int GTM = 64, GTN = 32, GK = 16;
constexpr int GWN = 16;          // columns per warp
constexpr int GEMM_THREADS = GTM / 32 * (GTN / GWN) * 32;
// shared pitches (doubles): the fragment loads of a half-warp (rows g = 0..3
// or 4..7, columns t = 0..3) fall in distinct banks: 2 (20 g + t) and
// 2 (36 t + g) mod 32 are distinct over the 16 lanes
constexpr int AS_LD = GK + 4;    // As[m][k]
constexpr int BS_LD = GTN + 4;   // Bs[k][n]
constexpr int AS_SIZE = GTM * AS_LD, BS_SIZE = GK * BS_LD;

// 16-byte global -> shared copy; zeros past the source size.
__device__ __forceinline__ void cp_async16(uint32_t dst, const double* src, int size) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(size) : "memory");
}

// c += a b, 16 x 8 x 8. Thread (g, t) = (lane / 4, lane % 4) holds a[i] at
// row g + 8 (i & 1), k t + 4 (i >> 1); b[i] at k t + 4 i, column g; c[i] at
// row g + 8 (i >> 1), column 2 t + (i & 1).
__device__ __forceinline__ void dmma(double (&c)[4], const double (&a)[4], const double (&b)[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

__global__ void __launch_bounds__(GEMM_THREADS, 6) dgemm_kernel(const __grid_constant__ GemmBatch b) {
    __shared__ __align__(16) double As[2 * AS_SIZE], Bs[2 * BS_SIZE];
    const int bid = blockIdx.x;
    int pi = 0;
#pragma unroll 1
    for (int q = 1; q < b.count; ++q)
        if (bid >= b.p[q].tile_start) pi = q;
    const GemmProb& P = b.p[pi];
    const int t = bid - P.tile_start;
    const int tm = t / P.tiles_n, tn = t - tm * P.tiles_n;
    const int row0 = tm * GTM, col0 = tn * GTN;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, tq = lane & 3;            // fragment row group, thread in group
    const int wm = warp % (GTM / 32) * 32, wn = warp / (GTM / 32) * GWN;
    pdl_wait();

    // Rows of A past M and columns of B past N repeat the last ones (nothing of
    // them is stored), so a copy's address costs a clamp and a multiply; past
    // K zeros are copied. Rows start on 16 bytes at an even pitch, so a copy
    // of two columns that starts inside a row stays inside it. A: 16 rows x 16 k
    // per pass of the threads; B: 8 k rows x 32 columns.
    static_assert(GEMM_THREADS == 128 && GK == 16 && GTN == 32, "the copies' shapes");
    const int ra = tid >> 3, ka = (tid & 7) * 2, kb = tid >> 4, nb = (tid & 15) * 2;
    const int alast = P.M - 1 - row0 - ra;
    const double* pa = P.A + (size_t)(row0 + ra) * P.lda + ka;
    const double* pb = P.B + (size_t)kb * P.ldb + min(col0 + nb, (P.N - 1) & ~1);
    const uint32_t sa = static_cast<uint32_t>(__cvta_generic_to_shared(As + ra * AS_LD + ka));
    const uint32_t sb = static_cast<uint32_t>(__cvta_generic_to_shared(Bs + kb * BS_LD + nb));
    auto load = [&](int k0, int buf) {
        const int size_a = max(0, min(2, P.K - k0 - ka)) * 8;
        const double* a = size_a ? pa + k0 : P.A;
        const int lda = size_a ? P.lda : 0;
#pragma unroll
        for (int i = 0; i < GTM / 16; ++i)
            cp_async16(sa + (buf * AS_SIZE + i * 16 * AS_LD) * 8, a + (ptrdiff_t)min(i * 16, alast) * lda, size_a);
        const double* b = pb + (size_t)k0 * P.ldb;
#pragma unroll
        for (int i = 0; i < GK / 8; ++i) {
            const bool in = k0 + kb + 8 * i < P.K;
            cp_async16(sb + (buf * BS_SIZE + i * 8 * BS_LD) * 8, in ? b + (ptrdiff_t)(8 * i) * P.ldb : P.B, in ? 16 : 0);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    double acc[2][GWN / 8][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < GWN / 8; ++j)
#pragma unroll
            for (int h = 0; h < 4; ++h) acc[i][j][h] = 0.0;

    const int nk = (P.K + GK - 1) / GK;
    load(0, 0);
    for (int kt = 0; kt < nk; ++kt) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();   // k-step kt is in; every warp is done with the other buffer
        if (kt + 1 < nk) load((kt + 1) * GK, (kt + 1) & 1);
        const double* as = As + (kt & 1) * AS_SIZE + (wm + g) * AS_LD + tq;
        const double* bs = Bs + (kt & 1) * BS_SIZE + tq * BS_LD + wn + g;
#pragma unroll
        for (int ks = 0; ks < GK; ks += 8) {
            double af[2][4], bf[GWN / 8][2];
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int h = 0; h < 4; ++h) af[i][h] = as[(i * 16 + (h & 1) * 8) * AS_LD + ks + (h >> 1) * 4];
#pragma unroll
            for (int j = 0; j < GWN / 8; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) bf[j][h] = bs[(ks + h * 4) * BS_LD + j * 8];
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < GWN / 8; ++j) dmma(acc[i][j], af[i], bf[j]);
        }
    }
    // accumulator (i, j, h): row wm + 16 i + g + 8 (h >> 1), column wn + 8 j +
    // 2 tq + (h & 1); a row's Lambda values are loaded together, ahead of its stores
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int row = row0 + wm + 8 * i + g, c0 = col0 + wn + 2 * tq;
        if (row >= P.M) continue;
        double l[GWN / 4];
        if (P.L)
#pragma unroll
            for (int u = 0; u < GWN / 4; ++u) {
                const int col = c0 + u / 2 * 8 + u % 2;
                l[u] = col < P.N ? __ldg(P.L + (size_t)row * P.ldl + col) : 0.0;
            }
#pragma unroll
        for (int u = 0; u < GWN / 4; ++u) {
            const int col = c0 + u / 2 * 8 + u % 2;
            if (col >= P.N) continue;
            double v = acc[i >> 1][u / 2][(i & 1) * 2 + u % 2];
            if (P.L) v *= l[u];
            P.C[(size_t)row * P.ldc + col] = v;
        }
    }
}

int launch_gemm(lc3d_ctx* c, GemmBatch& b, cudaStream_t s) {
    int tiles = 0;
    for (int q = 0; q < b.count; ++q) {
        GemmProb& p = b.p[q];
        p.tiles_n = (p.N + GTN - 1) / GTN;
        p.tile_start = tiles;
        tiles += ((p.M + GTM - 1) / GTM) * p.tiles_n;
    }
    if (tiles == 0) return LC3D_OK;
    ProfScope ps(c, LC3D_STAGE_TRANSFORM, s);
    LC3D_CUDA_TRY(launch_pdl(dgemm_kernel, dim3(tiles), dim3(GEMM_THREADS), 0, s, b));
    LC3D_CUDA_TRY(cudaGetLastError());
    return LC3D_OK;
}

// sin(pi r / L) for integer r, with the argument reduced to [0, pi/2].
double sin_pi_frac(long long r, long long L) {
    r %= 2 * L;
    if (r < 0) r += 2 * L;
    double sign = 1;
    if (r >= L) { r -= L; sign = -1; }
    if (2 * r > L) r = L - r;
    return sign * std::sin(M_PI * (double)r / (double)L);
}

// Half-size matrices of a transform type, by parity q (0 even, 1 odd) of the
// frequency: forth[k][n] = T[2 k + q][n], back[n][k] = T[n][2 k + q], and
// their transposes, all n_q x n_q at a pitch of whole lines.
struct HalfMats {
    double *forth, *forth_t, *back, *back_t;
};

struct DenseState {
    HalfMats m[2][2];       // [type][parity]
    double* lam[4];         // by type0 * 2 + type1, sorted by parity
};

// Size of parity q's half of a transform of `n` points (odd).
int half(int n, int q) { return q ? n / 2 : n / 2 + 1; }

int mat_pitch(int n) { return (n + 15) & ~15; }

}  // namespace

int dense_init(lc3d_ctx* c) {
    DenseState* d = new DenseState();
    c->dense = d;
    const int N = c->N;
    const long long L = N - 1;
    for (int type = 0; type < 2; ++type)
        for (int q = 0; q < 2; ++q) {
            const int n = half(N - 2 * type, q);
            // T[k][x]: 2 sin(pi (k+1)(x+1) / L), or c_x cos(pi k x / L) with
            // cos(pi r / L) = sin(pi (2 r + L) / (2 L))
            auto T = [&](long long k, long long x) {
                if (type) return 2 * sin_pi_frac((k + 1) * (x + 1), L);
                const long long r = (k * x) % (2 * L);
                return (x == 0 || x == L ? 1.0 : 2.0) * sin_pi_frac(2 * r + L, 2 * L);
            };
            const int ld = mat_pitch(n);
            const size_t nn = (size_t)n * ld;
            std::vector<double> h((type ? 2 : 4) * nn, 0.0);   // the DST-I matrix is symmetric: back = forth_t
            for (int k = 0; k < n; ++k)
                for (int x = 0; x < n; ++x) {
                    const double f = T(2 * k + q, x);
                    h[(size_t)k * ld + x] = f;
                    h[nn + (size_t)x * ld + k] = f;
                    if (type) continue;
                    const double b = T(x, 2 * k + q);
                    h[2 * nn + (size_t)x * ld + k] = b;
                    h[3 * nn + (size_t)k * ld + x] = b;
                }
            HalfMats& m = d->m[type][q];
            LC3D_CUDA_TRY(cudaMalloc(&m.forth, h.size() * sizeof(double)));
            LC3D_CUDA_TRY(cudaMemcpy(m.forth, h.data(), h.size() * sizeof(double), cudaMemcpyHostToDevice));
            m.forth_t = m.forth + nn;
            m.back = type ? m.forth_t : m.forth + 2 * nn;
            m.back_t = type ? m.forth : m.forth + 3 * nn;
        }
    const double* src[4] = {c->lam_neu, c->lam_mixT, c->lam_mix, c->lam_dir};
    for (int k = 0; k < 4; ++k) {
        const int rows = N - 2 * (k >> 1), cols = N - 2 * (k & 1);
        const int width = folded_width(cols);
        LC3D_CUDA_TRY(cudaMalloc(&d->lam[k], (size_t)rows * width * sizeof(double)));
        lam_parity_kernel<<<dim3((width + 127) / 128, rows), 128>>>(src[k], rows, cols, d->lam[k]);
        LC3D_CUDA_TRY(cudaGetLastError());
    }
    fields_drop_lam(c);   // this state has its own, sorted by parity
    return LC3D_OK;
}

void dense_free(lc3d_ctx* c) {
    DenseState* d = static_cast<DenseState*>(c->dense);
    if (!d) return;
    for (auto& type : d->m)
        for (HalfMats& m : type)
            if (m.forth) cudaFree(m.forth);
    for (double* l : d->lam)
        if (l) cudaFree(l);
    delete d;
    c->dense = nullptr;
}

int dense_solve(lc3d_ctx* c, const DenseDesc* desc, int count, cudaStream_t s) {
    const DenseState* d = static_cast<const DenseState*>(c->dense);
    const int N = c->N, ld = fft64_pitch(N);   // t1, t2: rows on whole lines
    const dim3 fold_grid(((N + 1) / 2 + 127) / 128, (N + 1) / 2, count);
    FoldArgs fa{};
    fa.ld_in = N;
    fa.ld_out = ld;
    for (int f = 0; f < count; ++f) {
        fa.rows[f] = N - 2 * desc[f].type0;
        fa.cols[f] = N - 2 * desc[f].type1;
        fa.in[f] = desc[f].rhs;
        fa.out[f] = desc[f].t2;
    }
    {
        ProfScope ps(c, LC3D_STAGE_TRANSFORM, s);
        LC3D_CUDA_TRY(launch_pdl(fold_kernel, fold_grid, dim3(128), 0, s, fa));
        LC3D_CUDA_TRY(cudaGetLastError());
    }
    for (int stage = 0; stage < 4; ++stage) {
        GemmBatch b;
        memset(&b, 0, sizeof(b));
        for (int f = 0; f < count; ++f) {
            const DenseDesc& e = desc[f];
            const int rows = fa.rows[f], cols = fa.cols[f];
            const bool right = stage == 0 || stage == 2, back = stage >= 2;
            for (int q = 0; q < 2; ++q) {
                GemmProb& p = b.p[b.count++];
                const double* in = right ? e.t2 : e.t1;
                double* out = right ? e.t1 : e.t2;
                if (right) {        // columns of parity q
                    const int n = half(cols, q), at = q * odd_at(cols);
                    const HalfMats& m = d->m[e.type1][q];
                    p.A = in + at; p.lda = ld;
                    p.B = back ? m.back_t : m.forth_t; p.ldb = mat_pitch(n);
                    p.C = out + at; p.ldc = ld;
                    p.M = rows; p.N = n; p.K = n;
                } else {            // rows of parity q
                    const int n = half(rows, q), at = q * half(rows, 0);
                    const HalfMats& m = d->m[e.type0][q];
                    p.A = back ? m.back : m.forth; p.lda = mat_pitch(n);
                    p.B = in + (size_t)at * ld; p.ldb = ld;
                    p.C = out + (size_t)at * ld; p.ldc = ld;
                    p.M = n; p.N = folded_width(cols); p.K = n;
                    if (!back) {
                        p.L = d->lam[e.type0 * 2 + e.type1] + (size_t)at * p.N;
                        p.ldl = p.N;
                    }
                }
            }
        }
        LC3D_TRY(launch_gemm(c, b, s));
    }
    fa.ld_in = ld;
    fa.ld_out = N;
    for (int f = 0; f < count; ++f) {
        fa.in[f] = desc[f].t2;
        fa.out[f] = desc[f].out;
    }
    ProfScope ps(c, LC3D_STAGE_TRANSFORM, s);
    LC3D_CUDA_TRY(launch_pdl(unfold_kernel, fold_grid, dim3(128), 0, s, fa));
    LC3D_CUDA_TRY(cudaGetLastError());
    return LC3D_OK;
}
