// Plasma particle kernels: field-free estimate, pusher with TSC field gather,
// coarse->fine interpolation with deterministic 9-point TSC deposition.
//
// Reference: lcode.py:369-391 (move_estimate_wo_fields), 396-449 (weights,
// interp9, deposit9), 576-689 (mix, coarse_to_fine, deposit_kernel,
// deposit), 704-823 (move_smart_kernel, move_smart).
//
// Deposition is deterministic. The reference adds every fine particle's 36
// contributions with float64 atomics in an unspecified order. Here every
// contribution c is split exactly into two integers,
//     c = hi * 2^-24 + lo * 2^-76 + (rounding below 2^-77),
// which are summed with 64-bit integer adds; integer addition is associative,
// so the sums do not depend on the order in which threads add them, and the
// final conversion rounds once. Each CTA owns a tile of 12 (or 4, 8, 16) fine
// lattice rows x 32 columns and accumulates into a shared-memory window
// placed on the bounding box of its particles' cells (float64 sums in a
// fixed order); particles outside the window (strongly displaced plasma) add
// straight to the global accumulators. The window is then flushed with 64-bit integer reductions into global memory, and a
// finalize pass converts to float64, adds the ion background and clears the
// accumulators for the next call.

#include <mutex>

#include "lc3d_internal.cuh"

namespace {

// ---------------------------------------------------------------------------
// TSC weights, lcode.py:396-418. Order MP 0P PP M0 00 P0 MM 0M PM.
// ---------------------------------------------------------------------------
struct Tsc {
    int i, j;
    double wxM, wx0, wxP, wyM, wy0, wyP;
};

// Centre cell (i, j) and offset from the cell centre, lcode.py:404-406.
// x / h correctly rounded from the reciprocal: q0 = x (1/h) is within an ulp,
// one Newton correction with the exact residual fma(-q0, h, x) rounds it.
__device__ __forceinline__ double div_h(double x, double h, double inv_h) {
    const double q0 = x * inv_h;
    return fma(fma(-q0, h, x), inv_h, q0);
}

// sqrt(S) and 1 / sqrt(S) without branches (the library's functions end each
// block of instructions with a test for their slow path, so chains of several
// particles, or of one particle's quotients, do not overlap): Goldschmidt's
// iteration for sqrt(S) and 1 / (2 sqrt(S)) from the hardware's approximation,
// both corrected by their exact residuals (Markstein). S normal and well
// inside the range: in_fast_range. With recip_fast and div_h 38 million random
// quotients by square roots all came out correctly rounded.
__device__ __forceinline__ void sqrt_fast(double S, double& g, double& inv) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(S));
    double h = .5 * y;
    g = S * y;
#pragma unroll
    for (int it = 0; it < 2; ++it) {
        const double e = fma(-g, h, .5);
        g = fma(g, e, g);
        h = fma(h, e, h);
    }
    g = fma(fma(-g, g, S), h, g);
    inv = h + h;
    inv = fma(inv, fma(-g, inv, 1.0), inv);
}
__device__ __forceinline__ bool in_fast_range(double S) { return S > 0x1p-900 && S < 0x1p900; }

// 1 / d by Newton's iteration, for a quotient x / d = div_h(x, d, recip_fast(d));
// d not 0.
__device__ __forceinline__ double recip_fast(double d) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
#pragma unroll
    for (int it = 0; it < 2; ++it) r = fma(r, fma(-d, r, 1.0), r);
    return r;
}

__device__ __forceinline__ void tsc_cell(double x, double y, int N, double h, double inv_h, int& i, int& j,
                                         double& xl, double& yl) {
    double x_h = div_h(x, h, inv_h) + .5, y_h = div_h(y, h, inv_h) + .5;
    double fx = floor(x_h), fy = floor(y_h);
    xl = x_h - fx - .5;
    yl = y_h - fy - .5;
    // out-of-range positions map to an invalid index without UB in the cast
    fx = fmin(fmax(fx, -1.0e6), 1.0e6);
    fy = fmin(fmax(fy, -1.0e6), 1.0e6);
    i = (int)fx + N / 2;
    j = (int)fy + N / 2;
}

// Quadratic-spline weights along one axis, lcode.py:410-412.
__device__ __forceinline__ void tsc_axis(double l, double& wM, double& w0, double& wP) {
    w0 = .75 - l * l;
    wP = (.5 + l) * (.5 + l) / 2;
    wM = (.5 - l) * (.5 - l) / 2;
}

__device__ __forceinline__ Tsc tsc_weights(double x, double y, int N, double h, double inv_h) {
    Tsc t;
    double xl, yl;
    tsc_cell(x, y, N, h, inv_h, t.i, t.j, xl, yl);
    tsc_axis(xl, t.wxM, t.wx0, t.wxP);
    tsc_axis(yl, t.wyM, t.wy0, t.wyP);
    return t;
}

__device__ __forceinline__ bool tsc_in_grid(const Tsc& t, int N) {
    return t.i >= 1 && t.i <= N - 2 && t.j >= 1 && t.j <= N - 2;
}

// interp9, lcode.py:421-430 (same summation order), in two halves: the
// nine values a field is read at, then their weighted sum. The pusher issues
// all six fields' gathers before any sum, so the 54 loads of a particle are
// in flight together (one round of memory latency instead of several:
// 0.0416 -> 0.0342 ms per xi step at 641^2).
__device__ __forceinline__ void gather9(const double* __restrict__ a, const Tsc& t, int N, double (&v)[9]) {
    const double* r0 = a + (size_t)(t.i - 1) * N + t.j;   // row i-1
    const double* r1 = r0 + N;
    const double* r2 = r1 + N;
    v[0] = r0[+1]; v[1] = r1[+1]; v[2] = r2[+1];
    v[3] = r0[0];  v[4] = r1[0];  v[5] = r2[0];
    v[6] = r0[-1]; v[7] = r1[-1]; v[8] = r2[-1];
}
__device__ __forceinline__ double sum9(const double (&v)[9], const Tsc& t) {
    return v[0] * (t.wxM * t.wyP) + v[1] * (t.wx0 * t.wyP) + v[2] * (t.wxP * t.wyP) +
           v[3] * (t.wxM * t.wy0) + v[4] * (t.wx0 * t.wy0) + v[5] * (t.wxP * t.wy0) +
           v[6] * (t.wxM * t.wyM) + v[7] * (t.wx0 * t.wyM) + v[8] * (t.wxP * t.wyM);
}

// ---------------------------------------------------------------------------
// Field-free estimate, lcode.py:369-391 (reflection with >= and <=).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void estimate_one(double m, double xi0, double yi0, double xo, double yo,
                                             double px, double py, double pz, double dxi, double rb,
                                             double& ex, double& ey) {
    double x = xi0 + xo, y = yi0 + yo;
    const double S = m * m + pz * pz + px * px + py * py;
    double gamma_f, inv;
    sqrt_fast(S, gamma_f, inv);
    const double d = gamma_f - pz;
    double vx, vy;
    if (in_fast_range(S) && d != 0) {   // 0: pz swamps the rest
        const double r = recip_fast(d);
        vx = div_h(px, d, r);
        vy = div_h(py, d, r);
    } else {
        const double gamma_m = sqrt(S);
        vx = px / (gamma_m - pz);
        vy = py / (gamma_m - pz);
    }
    x += vx * dxi;
    y += vy * dxi;
    if (x >= +rb) x = +2 * rb - x;
    if (x <= -rb) x = -2 * rb - x;
    if (y >= +rb) y = +2 * rb - y;
    if (y <= -rb) y = -2 * rb - y;
    ex = x - xi0;
    ey = y - yi0;
}

__global__ void __launch_bounds__(256) move_estimate_kernel(EstimateArgs a) {
    pdl_wait();
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= a.n) return;
    double ex, ey;
    estimate_one(a.m[k], a.x_init[k], a.y_init[k], a.x_prev[k], a.y_prev[k], a.px[k], a.py[k],
                 a.pz[k], a.dxi, a.rb, ex, ey);
    a.out_x[k] = ex;
    a.out_y[k] = ey;
}

// One coarse particle's seven deposit inputs as 64 contiguous bytes, so that
// the deposition gathers a coarse neighbour with four 16-byte loads instead
// of seven scattered 8-byte ones.
__device__ __forceinline__ void store_packed(double* p, double x, double y, double m, double q, double px,
                                             double py, double pz) {
    double2* p2 = reinterpret_cast<double2*>(p);
    p2[0] = make_double2(x, y);
    p2[1] = make_double2(m, q);
    p2[2] = make_double2(px, py);
    p2[3] = make_double2(pz, 0.0);
}

// The momentum push, lcode.py:745-780 (the float64 step kernel of 161^2 spends
// its time in this chain: 80.1 -> 79.0 us per xi step without the branches, 81^2
// 74 -> 69, 641^2 363 -> 361): two passes from the old momenta in the
// gathered fields, then the velocity of the half-way momenta. FAST: without
// branches (sqrt_fast); returns false if a square root left its range or the
// last quotients' denominator is 0 (1 - vz = 0 makes the next square root NaN).
struct Push {
    double px, py, pz, dpx, dpy, dpz, vx, vy;   // half-way momenta, changes, dx / dxi, dy / dxi
};
template <bool FAST>
__device__ __forceinline__ bool push(double m, double q, double dxi, double opx, double opy, double opz, const double (&F)[6],
                                     Push& o) {
    bool ok = true;
    double px = opx, py = opy, pz = opz;
#pragma unroll
    for (int it = 0; it < 3; ++it) {
        const double S = m * m + pz * pz + px * px + py * py;
        double gamma_m, inv = 0;
        if (FAST) {
            ok = ok && in_fast_range(S);
            sqrt_fast(S, gamma_m, inv);
        } else {
            gamma_m = sqrt(S);
        }
        auto over_gamma = [&](double x) { return FAST ? div_h(x, gamma_m, inv) : x / gamma_m; };
        if (it == 2) {
            const double d = gamma_m - pz;
            if (FAST) {
                ok = ok && d != 0;   // 0: pz swamps the rest
                const double r = recip_fast(d);
                o.vx = div_h(px, d, r);
                o.vy = div_h(py, d, r);
            } else {
                o.vx = px / d;
                o.vy = py / d;
            }
            break;
        }
        const double vx = over_gamma(px), vy = over_gamma(py), vz = over_gamma(pz);
        const double d = 1 - vz;
        const double factor_1 = FAST ? div_h(q * dxi, d, recip_fast(d)) : q * dxi / d;
        o.dpx = factor_1 * (F[0] + vy * F[5] - vz * F[4]);
        o.dpy = factor_1 * (F[1] - vx * F[5] + vz * F[3]);
        o.dpz = factor_1 * (F[2] + vx * F[4] - vy * F[3]);
        px = opx + o.dpx / 2;
        py = opy + o.dpy / 2;
        pz = opz + o.dpz / 2;
    }
    o.px = px;
    o.py = py;
    o.pz = pz;
    return ok;
}

// ---------------------------------------------------------------------------
// Pusher, lcode.py:704-793. One thread per coarse particle. With est_x ==
// NULL the field-free estimate of lcode.py:369-391 is computed inline (the
// predictor pass of step()).
// ---------------------------------------------------------------------------
#ifndef LC3D_MOVE_THREADS
#define LC3D_MOVE_THREADS 64    // the gathers in flight take ~150 registers a thread: small CTAs keep
#endif                          // 42,025 particles (641^2) in one wave (64 measured a little ahead of 128)
__global__ void __launch_bounds__(LC3D_MOVE_THREADS, 1) move_smart_kernel(MoveArgs a) {
    pdl_wait();
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= a.n) return;
    const double m = a.m[k], q = a.q[k];
    const double xi0 = a.x_init[k], yi0 = a.y_init[k];
    const double opx = a.px_prev[k], opy = a.py_prev[k], opz = a.pz_prev[k];
    double x_offt = a.x_prev[k], y_offt = a.y_prev[k];
    double ex, ey;
    if (a.est_x) {
        ex = a.est_x[k];
        ey = a.est_y[k];
    } else {
        estimate_one(m, xi0, yi0, x_offt, y_offt, opx, opy, opz, a.dxi, a.rb, ex, ey);
    }
    double x_half = xi0 + (x_offt + ex) / 2;
    double y_half = yi0 + (y_offt + ey) / 2;
    Tsc t = tsc_weights(x_half, y_half, a.N, a.h, a.inv_h);
    if (!tsc_in_grid(t, a.N)) {
        // the reference would read out of bounds here; flag and keep prev
        raise_flag(a.err, LC3D_FLAG_WINDOW);
        a.out_x[k] = x_offt;
        a.out_y[k] = y_offt;
        a.out_px[k] = opx;
        a.out_py[k] = opy;
        a.out_pz[k] = opz;
        if (a.out_packed) store_packed(a.out_packed + 8 * (size_t)k, x_offt, y_offt, m, q, opx, opy, opz);
        return;
    }
    double g[6][9];
#pragma unroll
    for (int f = 0; f < 6; ++f) gather9(a.F[f], t, a.N, g[f]);
    double F[6];   // Ex Ey Ez Bx By Bz
#pragma unroll
    for (int f = 0; f < 6; ++f) F[f] = sum9(g[f], t);
    Push o;
    if (!push<true>(m, q, a.dxi, opx, opy, opz, F, o)) push<false>(m, q, a.dxi, opx, opy, opz, F, o);
    x_offt += o.vx * a.dxi;
    y_offt += o.vy * a.dxi;
    double px = opx + o.dpx, py = opy + o.dpy;
    const double pz = opz + o.dpz;

    const double rb = a.rb;
    double x = xi0 + x_offt, y = yi0 + y_offt;
    if (x > +rb) { x = +2 * rb - x; x_offt = x - xi0; px = -px; }
    if (x < -rb) { x = -2 * rb - x; x_offt = x - xi0; px = -px; }
    if (y > +rb) { y = +2 * rb - y; y_offt = y - yi0; py = -py; }
    if (y < -rb) { y = -2 * rb - y; y_offt = y - yi0; py = -py; }
    a.out_x[k] = x_offt;
    a.out_y[k] = y_offt;
    a.out_px[k] = px;
    a.out_py[k] = py;
    a.out_pz[k] = pz;
    if (a.out_packed) store_packed(a.out_packed + 8 * (size_t)k, x_offt, y_offt, m, q, px, py, pz);
}

// ---------------------------------------------------------------------------
// Exact fixed-point split of a contribution.
// hi = round(c * 2^24) through the 1.5*2^28 magic constant (valid for
// |c| < 2^27); r = c - hi*2^-24 is exact and |r| <= 2^-25, so
// lo = round(r * 2^76) through 1.5*2^-24. The bit-pattern difference of two
// doubles in the same (or the adjacent upper) binade counts ulps exactly.
// ---------------------------------------------------------------------------
constexpr double FX_MAX = 0x1p+27;

__device__ __forceinline__ void fx_split(double c, long long& hi, long long& lo) {
    const double MH = 0x1.8p+28;                      // 1.5 * 2^28
    const double ML = 0x1.8p-24;                      // 1.5 * 2^-24
    double t = c + MH;
    hi = __double_as_longlong(t) - __double_as_longlong(MH);
    double r = c - (t - MH);
    double t2 = r + ML;
    lo = __double_as_longlong(t2) - __double_as_longlong(ML);
}

// One fine particle: coarse->fine mix (lcode.py:591-621) and the deposit
// quantities (lcode.py:651-655).
struct FineParticle {
    double x, y, dro, djx, djy, djz;
};

// Deposit quantities from the mixed coarse values (lcode.py:651-655).
__device__ __forceinline__ void particle_values(FineParticle& p, double m, double q, double px, double py,
                                                double pz) {
    const double gamma_m = sqrt(m * m + px * px + py * py + pz * pz);
    // the two quotients by gamma_m from one reciprocal, each corrected by
    // its exact residual (div_h): the reference's divisions, one division
    // sequence fewer per particle (the algebraically equal single division
    // q / (gamma_m - pz) measured only 0.5 % faster and departs from the
    // reference's rounding)
    const double inv_g = 1.0 / gamma_m;
    p.dro = q / (1 - div_h(pz, gamma_m, inv_g));
    const double dro_g = div_h(p.dro, gamma_m, inv_g);
    p.djx = px * dro_g;
    p.djy = py * dro_g;
    p.djz = pz * dro_g;
}

// particle_values without branches, so that a thread's particles overlap
// (phase 1 of the deposition took 43 of 83 us with the library's functions).
// Returns false where the caller has to take particle_values.
__device__ __forceinline__ bool particle_values_fast(FineParticle& p, double m, double q, double px, double py,
                                                     double pz) {
    const double S = m * m + px * px + py * py + pz * pz;
    double g, inv;
    sqrt_fast(S, g, inv);
    const double d = 1 - div_h(pz, g, inv);
    p.dro = div_h(q, d, recip_fast(d));
    const double dro_g = div_h(p.dro, g, inv);
    p.djx = px * dro_g;
    p.djy = py * dro_g;
    p.djz = pz * dro_g;
    return in_fast_range(S);
}

// The cell of one coordinate and the offset from its centre (tsc_cell): the
// same floor, through the rounding of x_h + 1.5 2^52, whose low word is the
// integer.
__device__ __forceinline__ int tsc_cell_1(double x, int N, double h, double inv_h, double& xl) {
    constexpr double M = 0x1.8p52;
    const double x_h = div_h(x, h, inv_h) + .5;
    const double t = x_h + M;
    const bool up = t - M > x_h;
    const double f = up ? (t - M) - 1.0 : t - M;
    xl = x_h - f - .5;
    return fabs(x_h) < 1.0e6 ? __double2loint(t) - (up ? 1 : 0) + N / 2 : -1;
}

__device__ __forceinline__ FineParticle fine_particle(const DepositArgs& a, int fi, int fj) {
    const double ipi = a.inf_prev[fi], ini = a.inf_next[fi];
    const double ipj = a.inf_prev[fj], inj = a.inf_next[fj];
    const double A = ipi * ipj, B = ipi * inj, C = ini * ipj, D = ini * inj;
    const int pi = a.idx_prev[fi], ni = a.idx_next[fi];
    const int pj = a.idx_prev[fj], nj = a.idx_next[fj];
    const int kA = pi * a.Nc + pj, kB = pi * a.Nc + nj, kC = ni * a.Nc + pj, kD = ni * a.Nc + nj;
    FineParticle p;
    if (a.packed) {   // the same values and arithmetic, four 16-byte loads per neighbour
        const double2* P2 = reinterpret_cast<const double2*>(a.packed);
        double2 w[4][4];
        const int ks[4] = {kA, kB, kC, kD};
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int h = 0; h < 4; ++h) w[c][h] = __ldg(P2 + 4 * (size_t)ks[c] + h);
#define LC3D_MIX4(h, comp) (A * w[0][h].comp + B * w[1][h].comp + C * w[2][h].comp + D * w[3][h].comp)
        p.x = a.fine_grid[fi] + LC3D_MIX4(0, x);
        p.y = a.fine_grid[fj] + LC3D_MIX4(0, y);
        particle_values(p, a.sf * LC3D_MIX4(1, x), a.sf * LC3D_MIX4(1, y), a.sf * LC3D_MIX4(2, x),
                        a.sf * LC3D_MIX4(2, y), a.sf * LC3D_MIX4(3, x));
#undef LC3D_MIX4
        return p;
    }
#define LC3D_MIX(arr) (A * __ldg(arr + kA) + B * __ldg(arr + kB) + C * __ldg(arr + kC) + D * __ldg(arr + kD))
    p.x = a.fine_grid[fi] + LC3D_MIX(a.x_offt);
    p.y = a.fine_grid[fj] + LC3D_MIX(a.y_offt);
    particle_values(p, a.sf * LC3D_MIX(a.m), a.sf * LC3D_MIX(a.q), a.sf * LC3D_MIX(a.px), a.sf * LC3D_MIX(a.py),
                    a.sf * LC3D_MIX(a.pz));
#undef LC3D_MIX
    return p;
}

__device__ __forceinline__ void fx_add(unsigned long long* hi_plane, unsigned long long* lo_plane, size_t cell,
                                       double c) {
    long long hi, lo;
    fx_split(c, hi, lo);
    atomicAdd(hi_plane + cell, (unsigned long long)hi);
    atomicAdd(lo_plane + cell, (unsigned long long)lo);
}

// ---------------------------------------------------------------------------
// Deposition kernel. A CTA deposits a tile of TI fine-lattice rows x 32
// columns, three rows per warp (one on small lattices).
//  1. As many fine particles per thread, one per row of its warp. Coarse->fine
//     mix in two separable passes (the equivalent formula noted beside the
//     reference's make_plasma, lcode.py:554-556): the warp first mixes the two
//     coarse rows of each fine row fi,
//         R[c] = inf_prev[fi] Q[prev_i][c] + inf_next[fi] Q[next_i][c],
//     for the coarse columns c its lanes use (7 quantities, a warp-private
//     table in shared memory); each lane then mixes two entries,
//     Q = inf_prev[fj] R[prev_j] + inf_next[fj] R[next_j]. A tile whose
//     columns span more than DEP_CMAX coarse columns (other coarseness /
//     fineness settings, or arbitrary virt_params) mixes per particle from
//     global memory (fine_particle). Then the deposit values
//     (lcode.py:651-655) and the TSC cell; cell offsets and values are staged
//     in shared memory.
//  2. One thread per cell (two or four with the fields split between them on
//     small lattices). Every particle sets its bit in its cell's masks
//     (one word per fine row, one bit per column), so a cell's thread meets
//     its particles in the order of the lattice, whatever the timing. It sums
//     their stencils, all four fields, into a 3 x 3 patch in registers: the
//     weights of a particle are computed once, and a patch never spans more
//     than one cell, however the lattice has moved against the grid. The
//     patches are added to a float64 window in nine barrier-separated steps,
//     one patch entry a step: no two threads write one cell in a step.
//  3. Each touched window cell is split once into fixed point and added to
//     the global accumulators. A tile whose cells are too many for one window
//     (rarefied plasma) takes up to four, one strip of rows after the other;
//     particles outside all of them add straight to the accumulators.
//
// Tiles start `a.fine_off` fine particles before the lattice origin: with an
// even fineness the fine index pairs (odd, even) of an undisturbed lattice
// share a cell, so no row or column of cells is split between tiles.
//
// Bound by instruction issue and latency, at 16 warps per SM (the patch's 72
// registers): 641^2, plasma displaced by several cells, 33.4 M warp
// instructions of which 10.9 M float64, issue 50 %, 62 us a launch. Summing
// 2 x 2 blocks of the lattice per (block, field) instead, with their weights
// once per field and 4 x 4 patches wherever a block straddles cells, took 45 M
// and 88 us. Per phase (us): lattice and row tables 13, particles 14, masks 5,
// sums over cells 18, window steps 7, flush 6. Five CTAs per SM (96
// registers, spills) measured 71 against 67, cells listed fullest first 67
// against 66.
// ---------------------------------------------------------------------------
constexpr int DEP_TW = 32;                  // fine columns of a tile, one per lane
constexpr int DEP_CMAX = 16;                // coarse columns the row tables hold
constexpr int DEP_CELLS = 256;              // cells with particles in a window
constexpr int DEP_SIDE = 32;                // ... their rows or columns at most
constexpr int DEP_STRIPS = 4;               // windows of a tile, one after the other (rarefied plasma)
constexpr int DEP_WIN = 352;                // window cells, (rows + 2) (columns + 2) <= 340

// Threads of a tile of `ti` rows, `rpw` of them per warp. 12 rows, three per
// warp: 384 particles on 128 threads, and at most 7 x 17 cells of an
// undisturbed lattice, one round of the threads (us per deposition with its
// finalize, 12 / 4 / 8 / 16 rows, plasma displaced by several cells: 641^2
// 69.5 / 93.5 / 76.6 / 85.4, 321^2 21.6 / 26.7 / 22.4 / 25.8).
__host__ __device__ constexpr int dep_threads(int ti, int rpw = 3) { return (ti + rpw - 1) / rpw * 32; }

// A lattice of few tiles leaves most of the chip idle, and what counts is how
// long one tile takes: four rows, one per warp (a row's particles are a chain
// of some 150 float64 instructions, three rows on a warp three times that on
// one float64 pipe), and a cell's fields split over up to four threads, since a
// cell holds fineness^2 particles one after the other. Up to 400 fine
// particles a side, where this shape and 12 rows meet (us per deposition with
// its finalize, this shape / 12 rows, plasma displaced by several cells:
// fineness 1: 161^2 11.4 / 18.6, 441^2 28.2 / 28.4; fineness 3: 121^2 9.9 /
// 11.6, 161^2 14.7 / 13.7; fineness 4: 81^2 9.2 / 13.7, 161^2 21.3 / 22.7). The
// threads of the 12-row tiles are fitted to fineness 2, and there the line is
// 240: 41^2 6.5 / 8.4, 81^2 8.0 / 10.8, 121^2 8.6 / 11.5; 161^2 is still ahead
// alone, 10.2 / 11.6, but in a batch, where other simulations fill the chip,
// its larger work shows: 8 simulations of 161^2 to 641^2 1292 us a step
// against 1266.
constexpr int DEP_SMALL_ROWS = 4;
// Threads per cell of that shape (1, 2 or 4), 0 where it does not apply. More
// threads cost more rounds of the window steps (us with 1 / 2 / 4: fineness 1,
// 161^2 11.4 / 11.7 / 13.7; fineness 2, 121^2 9.2 / 8.6 / 9.9; fineness 4,
// 81^2 10.7 / 10.0 / 9.2).
__host__ __device__ inline int dep_small(const DepositArgs& a) {
    return a.Nf > (a.fineness == 2 ? 240 : 400) ? 0 : a.fineness <= 1 ? 1 : a.fineness <= 3 ? 2 : 4;
}

// Staged particle of column `col` of a row: even columns, then odd ones, at a
// pitch of 36. Lanes of neighbouring cells read every other column, lanes of a
// warp write all of them; both touch distinct banks.
constexpr int DEP_ROW = 36;
__device__ __forceinline__ int dep_slot(int col) { return (col >> 1) + (col & 1) * 20; }

template <int TI>
__host__ __device__ constexpr size_t dep_table_words() {   // double2 words: the row tables, then the window
    constexpr size_t table = (size_t)TI * DEP_CMAX * 4, win = 2 * DEP_WIN;
    return table > win ? table : win;
}
template <int TI>
constexpr size_t dep_smem() {
    return ((size_t)TI * DEP_ROW * 3 + dep_table_words<TI>()) * sizeof(double2)   // (xl, yl), (ro, jx), (jy, jz); table
           + (TI + 1) * DEP_CELLS * sizeof(unsigned);                            // masks, rows in use
}

// Two of the seven coarse quantities of coarse particle k as a pair: h = 0
// (x_offt, y_offt), 1 (m, q), 2 (px, py), 3 (pz, 0).
__device__ __forceinline__ double2 coarse_pair(const DepositArgs& a, int k, int h) {
    if (a.packed) return __ldg(reinterpret_cast<const double2*>(a.packed) + 4 * (size_t)k + h);
    switch (h) {
        case 0: return make_double2(__ldg(a.x_offt + k), __ldg(a.y_offt + k));
        case 1: return make_double2(__ldg(a.m + k), __ldg(a.q + k));
        case 2: return make_double2(__ldg(a.px + k), __ldg(a.py + k));
        default: return make_double2(__ldg(a.pz + k), 0.0);
    }
}

// TI fine rows, RPW of them per warp, FS threads per cell.
template <int TI, int RPW = 3, int FS = 1>
__device__ __forceinline__ void deposit_tile(const DepositArgs& a, int tile_x, int tile_y) {
    constexpr int T = dep_threads(TI, RPW), P = TI * DEP_ROW;
    static_assert(TI <= 32, "masks of 32 bits");
    extern __shared__ __align__(16) double smem_f64[];
    double2* s_pos = reinterpret_cast<double2*>(smem_f64);               // [P] cell offsets
    double2* s_v01 = s_pos + P;                                          // [P] ro, jx
    double2* s_v23 = s_v01 + P;                                          // [P] jy, jz
    double2* s_R = s_v23 + P;                                            // [TI][DEP_CMAX][4]; then the window
    double2* s_win = s_R;                                                // [2][DEP_WIN]: ro, jx; jy, jz
    unsigned* s_mask = reinterpret_cast<unsigned*>(s_R + dep_table_words<TI>());   // [TI][DEP_CELLS]
    unsigned* s_rows = s_mask + TI * DEP_CELLS;                          // [DEP_CELLS]
    __shared__ int s_bb[4];                                              // imin imax jmin jmax
    const int t = threadIdx.x, lane = t & 31, row0 = (t >> 5) * RPW;
    if (t == 0) {
        s_bb[0] = s_bb[2] = 1 << 30;
        s_bb[1] = s_bb[3] = -(1 << 30);
    }
    {
        uint4* z = reinterpret_cast<uint4*>(s_mask);
        for (int w = t; w < (TI + 1) * DEP_CELLS / 4; w += T) z[w] = make_uint4(0u, 0u, 0u, 0u);
    }
    const int N = a.N;
    const size_t NN = a.plane;
    pdl_wait();   // global memory from here on

    // ---- phase 1 ----
    const int fi0 = tile_y * TI - a.fine_off + row0, fj = tile_x * DEP_TW - a.fine_off + lane;
    const bool col_ok = fj >= 0 && fj < a.Nf;
    int pi[RPW], ni[RPW], pj = 0, nj = 0;
    double ipi[RPW], ini[RPW], fgi[RPW], ipj = 0, inj = 0, fgj = 0;
    bool row_ok[RPW];
#pragma unroll
    for (int u = 0; u < RPW; ++u) {
        const int fi = fi0 + u;
        row_ok[u] = row0 + u < TI && fi >= 0 && fi < a.Nf;
        pi[u] = ni[u] = 0;
        ipi[u] = ini[u] = fgi[u] = 0;
        if (row_ok[u]) {
            pi[u] = a.idx_prev[fi];
            ni[u] = a.idx_next[fi];
            ipi[u] = a.inf_prev[fi];
            ini[u] = a.inf_next[fi];
            fgi[u] = a.fine_grid[fi];
        }
    }
    if (col_ok) {
        pj = a.idx_prev[fj];
        nj = a.idx_next[fj];
        ipj = a.inf_prev[fj];
        inj = a.inf_next[fj];
        fgj = a.fine_grid[fj];
    }
    const bool col_idx = pj >= 0 && pj < a.Nc && nj >= 0 && nj < a.Nc;
    // the coarse columns of the tile (the same in every warp)
    const int c0 = __reduce_min_sync(0xffffffffu, col_ok ? (col_idx ? min(pj, nj) : -(1 << 30)) : 1 << 30);
    const int c1 = __reduce_max_sync(0xffffffffu, col_ok ? (col_idx ? max(pj, nj) : 1 << 30) : -(1 << 30));
    const int nc = c1 - c0 + 1;
    const bool staged = c0 >= 0 && nc >= 1 && nc <= DEP_CMAX;
    bool ok[RPW];
#pragma unroll
    for (int u = 0; u < RPW; ++u) {
        const bool idx = pi[u] >= 0 && pi[u] < a.Nc && ni[u] >= 0 && ni[u] < a.Nc;
        if (row_ok[u] && col_ok && !(idx && col_idx)) raise_flag(a.err, LC3D_FLAG_WINDOW);
        if (!idx) pi[u] = ni[u] = 0;   // nobody uses that row of the table
        ok[u] = row_ok[u] && col_ok && idx && col_idx;
    }
    double2* R = s_R + row0 * DEP_CMAX * 4;
    if (staged) {
        for (int it = lane; it < nc * 4; it += 32) {
            const int jc = it >> 2, h = it & 3;
            double2 qp[RPW], qn[RPW];
#pragma unroll
            for (int u = 0; u < RPW; ++u) {
                if (row0 + u >= TI) continue;
                qp[u] = coarse_pair(a, pi[u] * a.Nc + c0 + jc, h);
                qn[u] = coarse_pair(a, ni[u] * a.Nc + c0 + jc, h);
            }
#pragma unroll
            for (int u = 0; u < RPW; ++u) {
                if (row0 + u >= TI) continue;
                R[u * DEP_CMAX * 4 + it] = make_double2(ipi[u] * qp[u].x + ini[u] * qn[u].x,
                                                        ipi[u] * qp[u].y + ini[u] * qn[u].y);
            }
        }
    }
    __syncwarp();
    int cell[RPW];   // i << 16 | j, or -1
    {
        const int op = (staged && col_ok ? pj - c0 : 0) * 4, on = (staged && col_ok ? nj - c0 : 0) * 4;
        FineParticle f[RPW];
        bool slow = !staged;
        double q[RPW][5];
        if (staged) {
#pragma unroll
            for (int u = 0; u < RPW; ++u) {
                const double2* Ru = R + (row0 + u < TI ? u : 0) * DEP_CMAX * 4;
                double2 w[4];
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const double2 rp = Ru[op + h], rn = Ru[on + h];
                    w[h] = make_double2(ipj * rp.x + inj * rn.x, ipj * rp.y + inj * rn.y);
                }
                f[u].x = fgi[u] + w[0].x;
                f[u].y = fgj + w[0].y;
                q[u][0] = a.sf * w[1].x;
                q[u][1] = a.sf * w[1].y;
                q[u][2] = a.sf * w[2].x;
                q[u][3] = a.sf * w[2].y;
                q[u][4] = a.sf * w[3].x;
            }
#pragma unroll
            for (int u = 0; u < RPW; ++u)
                if (!particle_values_fast(f[u], q[u][0], q[u][1], q[u][2], q[u][3], q[u][4]) && ok[u]) slow = true;
        }
        if (slow) {
#pragma unroll 1
            for (int u = 0; u < RPW; ++u)
                if (u == 0 ? ok[0] : u == 1 ? ok[1] : ok[2]) {
                    const FineParticle g = fine_particle(a, fi0 + u, fj);
#pragma unroll
                    for (int k = 0; k < RPW; ++k)
                        if (k == u) f[k] = g;
                }
        }
#pragma unroll
        for (int u = 0; u < RPW; ++u) {
            double xl, yl;
            const int i = tsc_cell_1(f[u].x, N, a.h, a.inv_h, xl), j = tsc_cell_1(f[u].y, N, a.h, a.inv_h, yl);
            const bool in = i >= 1 && i <= N - 2 && j >= 1 && j <= N - 2;
            // also false for NaN
            const bool fin = fabs(f[u].dro) < FX_MAX && fabs(f[u].djx) < FX_MAX && fabs(f[u].djy) < FX_MAX &&
                             fabs(f[u].djz) < FX_MAX;
            if (ok[u] && !in) raise_flag(a.err, LC3D_FLAG_WINDOW);
            if (ok[u] && in && !fin) raise_flag(a.err, LC3D_FLAG_NONFINITE);
            cell[u] = ok[u] && in && fin ? (i << 16) | j : -1;
            if (cell[u] >= 0) {
                const int k = (row0 + u) * DEP_ROW + dep_slot(lane);
                s_pos[k] = make_double2(xl, yl);
                s_v01[k] = make_double2(f[u].dro, f[u].djx);
                s_v23[k] = make_double2(f[u].djy, f[u].djz);
            }
        }
    }
    int imin = 1 << 30, imax = -(1 << 30), jmin = 1 << 30, jmax = -(1 << 30);
#pragma unroll
    for (int u = 0; u < RPW; ++u) {
        if (cell[u] < 0) continue;
        const int i = cell[u] >> 16, j = cell[u] & 0xffff;
        imin = min(imin, i);
        imax = max(imax, i);
        jmin = min(jmin, j);
        jmax = max(jmax, j);
    }
    imin = __reduce_min_sync(0xffffffffu, imin);
    imax = __reduce_max_sync(0xffffffffu, imax);
    jmin = __reduce_min_sync(0xffffffffu, jmin);
    jmax = __reduce_max_sync(0xffffffffu, jmax);
    // thread 0's empty bounding box is there before any warp adds to it. Here,
    // beside the next barrier, where the warps wait for the last one's phase 1
    // anyway
    __syncthreads();
    if (lane == 0 && imin <= imax) {
        atomicMin(&s_bb[0], imin);
        atomicMax(&s_bb[1], imax);
        atomicMin(&s_bb[2], jmin);
        atomicMax(&s_bb[3], jmax);
    }
    __syncthreads();   // the bounding box; the row tables are done with
    if (s_bb[0] > s_bb[1]) return;   // no particle (uniform)
    const int oj = s_bb[2], mj = min(s_bb[3] - oj + 1, DEP_SIDE);   // the first column of cells with particles, columns
    // quotients of small integers: (a + 0.5) / b lies at least 0.5 / b from an
    // integer, more than the float rounding
    const float inv_mj = 1.0f / (float)mj;
    const int strip_rows = min(DEP_SIDE, __float2int_rz((DEP_CELLS + 0.5f) * inv_mj)), wj = mj + 2;
    const int strips = min(__float2int_rz(((float)(s_bb[1] - s_bb[0]) + 0.5f) / (float)strip_rows) + 1, DEP_STRIPS);
    for (int strip = 0; strip < strips; ++strip) {
        // this window's cells with particles: mi rows from oi, mj columns from
        // oj; the window holds one cell more on each side
        const int oi = s_bb[0] + strip * strip_rows, mi = min(s_bb[1] - oi + 1, strip_rows);
        const int nwin = (mi + 2) * wj, ncell = mi * mj;
        for (int w = t; w < nwin; w += T)
            s_win[w] = s_win[DEP_WIN + w] = make_double2(0.0, 0.0);
        if (strip) {   // the first window's masks were cleared above
            uint4* z = reinterpret_cast<uint4*>(s_mask);
            for (int w = t; w < (TI + 1) * DEP_CELLS / 4; w += T) z[w] = make_uint4(0u, 0u, 0u, 0u);
            __syncthreads();
        }
#pragma unroll
        for (int u = 0; u < RPW; ++u) {
            if (cell[u] < 0) continue;
            const int row = row0 + u, i = (cell[u] >> 16) - oi, j = (cell[u] & 0xffff) - oj;
            if (i >= 0 && i < mi && j < mj) {
                const int c = i * mj + j;
                atomicOr(&s_mask[row * DEP_CELLS + c], 1u << lane);
                atomicOr(&s_rows[c], 1u << row);
            } else if (strip == 0 && (j >= mj || i >= strips * strip_rows)) {   // in no window
                const int k = row * DEP_ROW + dep_slot(lane);
                unsigned long long* g = a.acc + (size_t)(oi + i - 1) * N + (oj + j - 1);
                double wx[3], wy[3];
                tsc_axis(s_pos[k].x, wx[0], wx[1], wx[2]);
                tsc_axis(s_pos[k].y, wy[0], wy[1], wy[2]);
#pragma unroll 1
                for (int f = 0; f < 4; ++f) {
                    const double v = f == 0 ? s_v01[k].x : f == 1 ? s_v01[k].y : f == 2 ? s_v23[k].x : s_v23[k].y;
#pragma unroll
                    for (int e = 0; e < 9; ++e)
                        fx_add(g + 2 * f * NN, g + (2 * f + 1) * NN, (size_t)(e / 3) * N + e % 3, v * (wx[e / 3] * wy[e % 3]));
                }
            }
        }
        __syncthreads();   // masks complete, window cleared

        // ---- phase 2 ----
        // One cell per thread written out (as the general form's FS = 1 it
        // measured 1 to 2 % slower: a run step at 161^2 77.6 us against 76.2).
        if constexpr (FS == 1) {
            for (int r0 = 0; r0 < ncell; r0 += T) {
                const int c = r0 + t;
                unsigned rows = c < ncell ? s_rows[c] : 0u, m = 0;
                const bool any = rows != 0;
                const unsigned* mk = s_mask + c;
                int base = 0;
                double acc[4][9];
#pragma unroll
                for (int f = 0; f < 4; ++f)
#pragma unroll
                    for (int e = 0; e < 9; ++e) acc[f][e] = 0.0;
                while (rows | m) {
                    if (!m) {
                        const int r = __ffs(rows) - 1;
                        rows &= rows - 1;
                        m = mk[r * DEP_CELLS];
                        base = r * DEP_ROW;
                    }
                    const int k = base + dep_slot(__ffs(m) - 1);
                    m &= m - 1;
                    const double2 pos = s_pos[k], v01 = s_v01[k], v23 = s_v23[k];
                    double wx[3], wy[3];
                    tsc_axis(pos.x, wx[0], wx[1], wx[2]);
                    tsc_axis(pos.y, wy[0], wy[1], wy[2]);
                    const double v[4] = {v01.x, v01.y, v23.x, v23.y};
#pragma unroll
                    for (int f = 0; f < 4; ++f)
#pragma unroll
                        for (int di = 0; di < 3; ++di) {
                            const double vx = v[f] * wx[di];
#pragma unroll
                            for (int dj = 0; dj < 3; ++dj) acc[f][di * 3 + dj] = fma(vx, wy[dj], acc[f][di * 3 + dj]);
                        }
                }
                const int ci = __float2int_rz(((float)c + 0.5f) * inv_mj), cj = c - ci * mj;
                double2* w = s_win + ci * wj + cj;
#pragma unroll
                for (int e = 0; e < 9; ++e) {
                    if (any) {
                        double2* we = w + (e / 3) * wj + e % 3;
                        const double2 x = we[0], y = we[DEP_WIN];
                        we[0] = make_double2(x.x + acc[0][e], x.y + acc[1][e]);
                        we[DEP_WIN] = make_double2(y.x + acc[2][e], y.y + acc[3][e]);
                    }
                    __syncthreads();
                }
            }
        } else {   // FS threads per cell, 4 / FS fields each
            constexpr int NF = 4 / FS;
            for (int r0 = 0; r0 < ncell * FS; r0 += T) {
                const int c = (r0 + t) / FS, f0 = (r0 + t) % FS * NF;   // cell, first field
                unsigned rows = c < ncell ? s_rows[c] : 0u, m = 0;
                const bool any = rows != 0;
                const unsigned* mk = s_mask + c;
                const double2* sv = s_v01 + (f0 >> 1) * P;
                int base = 0;
                double acc[NF][9];
#pragma unroll
                for (int f = 0; f < NF; ++f)
#pragma unroll
                    for (int e = 0; e < 9; ++e) acc[f][e] = 0.0;
                while (rows | m) {
                    if (!m) {
                        const int r = __ffs(rows) - 1;
                        rows &= rows - 1;
                        m = mk[r * DEP_CELLS];
                        base = r * DEP_ROW;
                    }
                    const int k = base + dep_slot(__ffs(m) - 1);
                    m &= m - 1;
                    const double2 pos = s_pos[k];
                    double v[NF];
                    if constexpr (NF == 1) {
                        v[0] = f0 & 1 ? sv[k].y : sv[k].x;
                    } else {
                        double2 x[NF / 2];
#pragma unroll
                        for (int h = 0; h < NF / 2; ++h) x[h] = sv[h * P + k];
#pragma unroll
                        for (int f = 0; f < NF; ++f) v[f] = f & 1 ? x[f / 2].y : x[f / 2].x;
                    }
                    double wx[3], wy[3];
                    tsc_axis(pos.x, wx[0], wx[1], wx[2]);
                    tsc_axis(pos.y, wy[0], wy[1], wy[2]);
#pragma unroll
                    for (int f = 0; f < NF; ++f)
#pragma unroll
                        for (int di = 0; di < 3; ++di) {
                            const double vx = v[f] * wx[di];
#pragma unroll
                            for (int dj = 0; dj < 3; ++dj) acc[f][di * 3 + dj] = fma(vx, wy[dj], acc[f][di * 3 + dj]);
                        }
                }
                const int ci = __float2int_rz(((float)c + 0.5f) * inv_mj), cj = c - ci * mj;
                double2* w = s_win + (f0 >> 1) * DEP_WIN + ci * wj + cj;
#pragma unroll
                for (int e = 0; e < 9; ++e) {
                    if (any) {
                        double2* we = w + (e / 3) * wj + e % 3;
                        if constexpr (NF == 1) {
                            double& x = f0 & 1 ? we->y : we->x;
                            x += acc[0][e];
                        } else {
                            double2 x[NF / 2];
#pragma unroll
                            for (int h = 0; h < NF / 2; ++h) x[h] = we[h * DEP_WIN];
#pragma unroll
                            for (int h = 0; h < NF / 2; ++h)
                                we[h * DEP_WIN] = make_double2(x[h].x + acc[2 * h][e], x[h].y + acc[2 * h + 1][e]);
                        }
                    }
                    __syncthreads();
                }
            }
        }

        // ---- phase 3: split each touched window cell once, add to global ----
        const float inv_wj = 1.0f / (float)wj;
        for (int w = t; w < nwin; w += T) {
            const int ci = __float2int_rz(((float)w + 0.5f) * inv_wj), cj = w - ci * wj;
            unsigned long long* g = a.acc + (size_t)(oi - 1 + ci) * N + (oj - 1 + cj);
            const double2 x = s_win[w], y = s_win[DEP_WIN + w];
            const double v[4] = {x.x, x.y, y.x, y.y};
#pragma unroll
            for (int f = 0; f < 4; ++f)
                if (v[f] != 0.0) fx_add(g + 2 * f * NN, g + (2 * f + 1) * NN, 0, v[f]);
        }
        if (strip + 1 < strips) __syncthreads();   // the window is read; the next one clears it
    }
}

// One tile per CTA: blockIdx.x / .y = tile column / row. 16 warps per SM, the
// split cells' smaller patches 24.
template <int TI, int RPW = 3, int FS = 1>
__global__ void __launch_bounds__(dep_threads(TI, RPW), (FS > 1 ? 768 : 512) / dep_threads(TI, RPW))
    deposit_kernel(DepositArgs a) {
    deposit_tile<TI, RPW, FS>(a, blockIdx.x, blockIdx.y);
}

// Depositions of several simulations in one launch: CTA b takes the tile
// b - cta_start[s] of simulation s (cta_start: prefix sums of the tile
// counts, n + 1 entries), whose arguments are args[s]. Each simulation's tiles
// have the shape a launch of its own would give them.
static_assert(dep_threads(LC3D_DEP_ROWS) == dep_threads(DEP_SMALL_ROWS, 1), "one CTA size for all simulations");
__global__ void __launch_bounds__(dep_threads(LC3D_DEP_ROWS), 512 / dep_threads(LC3D_DEP_ROWS))
    deposit_multi_kernel(const DepositArgs* __restrict__ args, const int* __restrict__ cta_start, int n) {
    __shared__ DepositArgs sa;
    __shared__ int s_sim;
    if (threadIdx.x == 0) {
        int lo = 0, hi = n - 1;   // the last s with cta_start[s] <= blockIdx.x
        while (lo < hi) {
            const int mid = (lo + hi + 1) / 2;
            if (cta_start[mid] <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
        }
        s_sim = lo;
    }
    __syncthreads();
    {
        static_assert(sizeof(DepositArgs) % 4 == 0, "copied as words");
        const int* src = reinterpret_cast<const int*>(args + s_sim);
        int* dst = reinterpret_cast<int*>(&sa);
        for (int w = threadIdx.x; w < (int)(sizeof(DepositArgs) / 4); w += blockDim.x) dst[w] = src[w];
    }
    __syncthreads();
    const int t = (int)blockIdx.x - cta_start[s_sim];
    const int ntx = (sa.Nf + sa.fine_off + DEP_TW - 1) / DEP_TW;
    switch (dep_small(sa)) {
        case 0: deposit_tile<LC3D_DEP_ROWS>(sa, t % ntx, t / ntx); break;
        case 1: deposit_tile<DEP_SMALL_ROWS, 1, 1>(sa, t % ntx, t / ntx); break;
        case 2: deposit_tile<DEP_SMALL_ROWS, 1, 2>(sa, t % ntx, t / ntx); break;
        default: deposit_tile<DEP_SMALL_ROWS, 1, 4>(sa, t % ntx, t / ntx); break;
    }
}

// Accumulators -> float64 (+ ion background), two cells per thread; the
// accumulators are cleared for the next deposition. All eight 16-byte
// accumulator loads of a thread are issued before any store (the clears
// could alias later loads for the compiler otherwise, serialising them);
// the float64 side uses 16-byte accesses when every array allows it.
__global__ void __launch_bounds__(256) deposit_finalize_kernel(DepositFinalizeArgs f) {
    pdl_wait();
    const int k = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
    if (k >= f.n) return;
    const size_t P = f.plane;
    unsigned long long* acc = f.acc;
    if (k + 1 < f.n) {
        ulonglong2 w[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) w[q] = __ldcg(reinterpret_cast<const ulonglong2*>(acc + q * P + k));
        double2 ri = make_double2(0.0, 0.0);
        if (f.ro_initial) {
            if (f.vec) {
                ri = __ldg(reinterpret_cast<const double2*>(f.ro_initial + k));
            } else {
                ri.x = __ldg(f.ro_initial + k);
                ri.y = __ldg(f.ro_initial + k + 1);
            }
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) __stcg(reinterpret_cast<ulonglong2*>(acc + q * P + k), make_ulonglong2(0ull, 0ull));
        double2 o[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
            o[q] = make_double2(fx_value((long long)w[2 * q].x, (long long)w[2 * q + 1].x),
                                fx_value((long long)w[2 * q].y, (long long)w[2 * q + 1].y));
        if (f.ro_initial) {
            o[0].x += ri.x;
            o[0].y += ri.y;
        }
        double* dst[4] = {f.ro, f.jx, f.jy, f.jz};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (f.vec) {
                *reinterpret_cast<double2*>(dst[q] + k) = o[q];
            } else {
                dst[q][k] = o[q].x;
                dst[q][k + 1] = o[q].y;
            }
        }
    } else {
        double out[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            unsigned long long* hp = acc + (2 * q) * P + k;
            unsigned long long* lp = acc + (2 * q + 1) * P + k;
            out[q] = fx_value((long long)*hp, (long long)*lp);
            *hp = 0ull;
            *lp = 0ull;
        }
        double ro = out[0];
        if (f.ro_initial) ro += f.ro_initial[k];
        f.ro[k] = ro;
        f.jx[k] = out[1];
        f.jy[k] = out[2];
        f.jz[k] = out[3];
    }
}

}  // namespace

int launch_move_estimate(const EstimateArgs& a, cudaStream_t s) {
    if (a.n <= 0) return LC3D_OK;
    LC3D_CUDA_TRY(launch_pdl(move_estimate_kernel, dim3((a.n + 255) / 256), dim3(256), 0, s, a));
    LC3D_CUDA_TRY(cudaGetLastError());
    return LC3D_OK;
}

int launch_move_smart(const MoveArgs& a, cudaStream_t s) {
    if (a.n <= 0) return LC3D_OK;
    LC3D_CUDA_TRY(launch_pdl(move_smart_kernel, dim3((a.n + LC3D_MOVE_THREADS - 1) / LC3D_MOVE_THREADS),
                             dim3(LC3D_MOVE_THREADS), 0, s, a));
    LC3D_CUDA_TRY(cudaGetLastError());
    return LC3D_OK;
}

namespace {

// Rows of a tile at its default shape.
int dep_default_rows(const DepositArgs& a) { return dep_small(a) ? DEP_SMALL_ROWS : LC3D_DEP_ROWS; }

template <int TI, int RPW = 3, int FS = 1>
int prepare_deposit() {
    LC3D_CUDA_TRY(cudaFuncSetAttribute(deposit_kernel<TI, RPW, FS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)dep_smem<TI>()));
    return LC3D_OK;
}

template <int TI, int RPW = 3, int FS = 1>
int launch_deposit(const DepositArgs& a, cudaStream_t s) {
    const dim3 grid((a.Nf + a.fine_off + DEP_TW - 1) / DEP_TW, (a.Nf + a.fine_off + TI - 1) / TI);
    LC3D_CUDA_TRY(launch_pdl(deposit_kernel<TI, RPW, FS>, grid, dim3(dep_threads(TI, RPW)), dep_smem<TI>(), s, a));
    LC3D_CUDA_TRY(cudaGetLastError());
    return LC3D_OK;
}

}  // namespace

int particles_prepare() {
    LC3D_TRY(prepare_deposit<4>());
    LC3D_TRY(prepare_deposit<8>());
    LC3D_TRY(prepare_deposit<LC3D_DEP_ROWS>());
    LC3D_TRY(prepare_deposit<16>());
    LC3D_TRY((prepare_deposit<DEP_SMALL_ROWS, 1, 1>()));
    LC3D_TRY((prepare_deposit<DEP_SMALL_ROWS, 1, 2>()));
    LC3D_TRY((prepare_deposit<DEP_SMALL_ROWS, 1, 4>()));
    LC3D_CUDA_TRY(cudaFuncSetAttribute(deposit_multi_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)dep_smem<LC3D_DEP_ROWS>()));
    return LC3D_OK;
}

// Tile origin of the deposition: with an even fineness the fine lattice
// (lcode.py:468-487) puts two particles per cell and axis, and the pairs of
// fine indices (odd, even) share a cell, so tiles start one particle early.
int deposit_fine_offset(int fineness) {
#ifdef LC3D_DEP_FORCE_OFF
    (void)fineness;
    return LC3D_DEP_FORCE_OFF;
#else
    return fineness % 2 == 0 ? 1 : 0;
#endif
}

int launch_deposit_main(const DepositArgs& a, cudaStream_t s) {
    if (a.Nf <= 0) return LC3D_OK;
    switch (a.tile_rows) {
        case 0: break;
        case 4: return launch_deposit<4>(a, s);
        case 8: return launch_deposit<8>(a, s);
        case 16: return launch_deposit<16>(a, s);
        default: return LC3D_ERR_PARAM;
    }
    switch (dep_small(a)) {
        case 0: return launch_deposit<LC3D_DEP_ROWS>(a, s);
        case 1: return launch_deposit<DEP_SMALL_ROWS, 1, 1>(a, s);
        case 2: return launch_deposit<DEP_SMALL_ROWS, 1, 2>(a, s);
        default: return launch_deposit<DEP_SMALL_ROWS, 1, 4>(a, s);
    }
}

// Tiles of one simulation's deposition at its default shape.
int deposit_multi_tiles(const DepositArgs& a) {
    const int rows = dep_default_rows(a);
    return ((a.Nf + a.fine_off + DEP_TW - 1) / DEP_TW) * ((a.Nf + a.fine_off + rows - 1) / rows);
}

int launch_deposit_multi(const DepositArgs* args_dev, const int* cta_start_dev, int n, int ctas, cudaStream_t s) {
    if (n <= 0 || ctas <= 0) return LC3D_OK;
    static_assert(dep_smem<LC3D_DEP_ROWS>() >= dep_smem<DEP_SMALL_ROWS>(), "room for either shape");
    deposit_multi_kernel<<<ctas, dep_threads(LC3D_DEP_ROWS), dep_smem<LC3D_DEP_ROWS>(), s>>>(args_dev, cta_start_dev, n);
    LC3D_CUDA_TRY(cudaGetLastError());
    return LC3D_OK;
}

int launch_deposit_finalize(const DepositFinalizeArgs& f_in, cudaStream_t s) {
    DepositFinalizeArgs f = f_in;
    const uintptr_t al = reinterpret_cast<uintptr_t>(f.ro) | reinterpret_cast<uintptr_t>(f.jx) |
                         reinterpret_cast<uintptr_t>(f.jy) | reinterpret_cast<uintptr_t>(f.jz) |
                         reinterpret_cast<uintptr_t>(f.ro_initial);
    f.vec = (al & 15) == 0;
    LC3D_CUDA_TRY(launch_pdl(deposit_finalize_kernel, dim3(((f.n + 1) / 2 + 255) / 256), dim3(256), 0, s, f));
    LC3D_CUDA_TRY(cudaGetLastError());
    return LC3D_OK;
}

// ---------------------------------------------------------------------------
// Deposition without any device allocation.
//
// Some callers cannot allocate device memory when they deposit: a host
// program that reserved the GPU's memory up front for its own pool and
// forbids further cudaMalloc calls, or code that must not call cudaMalloc
// because it synchronises the device (a latency-critical loop) or is not
// allowed at all (while a CUDA graph is being captured). Creating a
// context (lc3d_create) allocates, so lc3d_deposit_noalloc takes every
// input from the caller and keeps its scratch -- the fixed-point
// accumulators and the error word -- in the file-scope device array below:
// 8 planes of LC3D_NOALLOC_MAX_GRID^2 64-bit words (6.6 MB for 321 x 321),
// which every GPU that loads this library holds until the process exits.
//
// Host code cannot use the array's name as a device address; the address
// is looked up once per device with cudaGetSymbolAddress (with that device
// current) on the first call made on that device, which also sets the
// kernel's shared-memory limit. That first call must therefore come before
// any stream capture. All calls share the array: each call clears the part
// it uses before depositing, and calls that overlap on the GPU (different
// streams, no ordering between them) race on it.
// ---------------------------------------------------------------------------

namespace {

constexpr size_t NOALLOC_PLANE =
    ((size_t)LC3D_NOALLOC_MAX_GRID * LC3D_NOALLOC_MAX_GRID + 31) / 32 * 32;
constexpr size_t NOALLOC_WORDS = DEP_WORDS_PER_CELL * NOALLOC_PLANE + 32;   // + error word (padded)

}  // namespace

static __device__ __align__(256) unsigned long long g_noalloc_scratch[NOALLOC_WORDS];

namespace {

constexpr int NOALLOC_MAX_DEVICES = 64;
std::mutex g_noalloc_mutex;
unsigned long long* g_noalloc_ptr[NOALLOC_MAX_DEVICES];

// Device address of g_noalloc_scratch on the current device (looked up once).
int noalloc_scratch(unsigned long long** out) {
    int dev = 0;
    LC3D_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) return LC3D_ERR_PARAM;
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[dev]) {
        void* p = nullptr;
        LC3D_CUDA_TRY(cudaGetSymbolAddress(&p, g_noalloc_scratch));
        LC3D_TRY(particles_prepare());
        g_noalloc_ptr[dev] = static_cast<unsigned long long*>(p);
    }
    *out = g_noalloc_ptr[dev];
    return LC3D_OK;
}

}  // namespace

extern "C" int lc3d_deposit_noalloc(const lc3d_params* p, const double* ro_initial, const double* x_offt,
                                    const double* y_offt, const double* m, const double* q, const double* px,
                                    const double* py, const double* pz, const double* influence_prev,
                                    const double* influence_next, const int32_t* indices_prev,
                                    const int32_t* indices_next, const double* fine_grid, double* out_ro,
                                    double* out_jx, double* out_jy, double* out_jz, void* stream) {
    int Nc = 0, Nf = 0;
    double rb = 0;
    LC3D_TRY(lc3d_sizes(p, &Nc, &Nf, &rb));
    if (p->grid_steps > LC3D_NOALLOC_MAX_GRID) return LC3D_ERR_SIZE;
    const void* req[] = {x_offt, y_offt, m, q, px, py, pz, influence_prev, influence_next,
                         indices_prev, indices_next, fine_grid, out_ro, out_jx, out_jy, out_jz};
    for (const void* r : req)
        if (!r) return LC3D_ERR_PARAM;
    unsigned long long* scratch = nullptr;
    LC3D_TRY(noalloc_scratch(&scratch));
    const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const int N = p->grid_steps;
    const size_t plane = ((size_t)N * N + 31) / 32 * 32;
    unsigned long long* err_word = scratch + DEP_WORDS_PER_CELL * NOALLOC_PLANE;
    // clear the accumulators this grid uses and the error word
    LC3D_CUDA_TRY(cudaMemsetAsync(scratch, 0, DEP_WORDS_PER_CELL * plane * sizeof(unsigned long long), s));
    LC3D_CUDA_TRY(cudaMemsetAsync(err_word, 0, sizeof(unsigned long long), s));
    const int c = p->plasma_coarseness, f = p->plasma_fineness;
    DepositArgs a{};
    a.x_offt = x_offt; a.y_offt = y_offt; a.m = m; a.q = q; a.px = px; a.py = py; a.pz = pz;
    a.inf_prev = influence_prev; a.inf_next = influence_next; a.fine_grid = fine_grid;
    a.idx_prev = indices_prev; a.idx_next = indices_next;
    a.acc = scratch;
    a.plane = plane;
    a.Nc = Nc; a.Nf = Nf; a.N = N;
    a.fineness = p->plasma_fineness;
    a.fine_off = deposit_fine_offset(p->plasma_fineness);
    a.h = p->grid_step_size;
    a.inv_h = 1.0 / p->grid_step_size;
    a.sf = 1.0 / ((double)(c * f) * (c * f));
    a.err = reinterpret_cast<unsigned*>(err_word);
    DepositFinalizeArgs fa{};
    fa.acc = scratch;
    fa.plane = plane;
    fa.ro_initial = ro_initial;
    fa.ro = out_ro; fa.jx = out_jx; fa.jy = out_jy; fa.jz = out_jz;
    fa.n = N * N;
    LC3D_TRY(launch_deposit_main(a, s));
    return launch_deposit_finalize(fa, s);
}
