// Float64 spectral field solves through shared-memory FFTs: three launches a
// solve for all fields, the step's field finalize in the last one.
//
// A solve is F = L (Lambda o (L X R)) R with L / R the DST-I or DCT-I along
// axis 0 / axis 1 (fields.cu; lcode.py:124-364). L and R act on different
// axes and commute, so the launches are
//     A:  rows of X along axis 1, written transposed
//     B:  rows of that along axis 0: transform, times Lambda, transform back,
//         written transposed
//     D:  rows of that along axis 1: F, with the Bz mean, Variant A and the
//         half-step averages applied as F is written (lcode.py:876-881)
// where the same four transforms as four passes needed a launch and a trip
// through memory each, and two launches more for the mean and the finalize.
//
// One transform. Two real rows a, b make z = a + i b, extended to length
// P = 2 (N - 1), z[P - j] = sigma z[j], sigma = +1 (DCT-I) or -1 (DST-I, whose
// result is -Im, Re). Z = FFT(z) has the same symmetry, and the first radix
// pass uses it (P = R1 M1, R1 even): with V_m the length-R1 DFT of the column
// z[j + r M1], r < R1,
//     y_m[j]      = W_P^(mj) V_m,      y_m[M1 - j] = sigma W_P^(-mj) V_(R1-m)
// so the columns j = 0 .. M1/2 give every y_m, and Z[m + R1 q] =
// FFT_M1(y_m)[q] is wanted for m = 0 .. R1/2 only: half the first pass and
// 9/16 (R1 = 16) of the others, no extension written or read. The way back is
// the transposed flow graph (decimation in time), which takes its input where
// the way forth leaves its output: B multiplies by Lambda in the registers of
// its middle radix pass, and no pass reorders anything. The order in which
// the kept frequencies lie in memory (`p` below) is the one the passes
// have them in; the Lambda table is laid out to match.
//
// A CTA transforms F = 4 or 8 pairs of rows, so that a transposed store
// fills whole sectors (F = 8: lines). Lanes run over the pairs in the passes
// that write transposed and over the columns in those that read or write rows.

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "lc3d_internal.cuh"

namespace {

constexpr int F64_THREADS = 512;          // at most
constexpr int MAX_MIDS = 6;

struct F64Plan {
    int N, L, P;
    int R1, M1;             // first radix, P / R1
    int nmid, rm[MAX_MIDS]; // radices between
    int RL;                 // last radix
    int nsub, ncol;         // R1 / 2 + 1 sub-transforms kept, M1 / 2 + 1 columns
    int NB, PB;             // butterflies of the last radix, the shared pitch between their elements (odd)
    int lf;                 // log2 of the row pairs per CTA
};

struct F64Field {
    const double* in;
    int ld_in, rows, type;  // rows of this launch; 0 DCT-I, 1 DST-I along them
    double* out;
    int ld_out;
    const double* lam;      // B: Lambda[position][row]
    int ld_lam;
    const double* sumw;     // B, Bz: weight of each row in the sum over the grid, or NULL
    double* partial;        // B, Bz: this field's sums per CTA; D: the same, to be read
    int npartial;
    const int* tab;         // A: row p of out at [q NB + b], or -1; D: column p of in, top bit: negated
    int border;             // axis 0 antisymmetric; A: the first grid row is not read; D: the first and last are zero
    int zero;               // D: a column of zeros in `in`
    const double* prev;     // D: step finalize
    double* avg;
    int variant_a;
    double inv_n;
    int cta_start;
};

struct F64Batch {
    F64Field f[6];
    int count;
    F64Plan p;
    const double2* tw;      // exp(-2 pi i m / P)
};

__device__ __forceinline__ double2 mk(double a, double b) { return make_double2(a, b); }
__device__ __forceinline__ double2 operator+(double2 a, double2 b) { return mk(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 operator-(double2 a, double2 b) { return mk(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 operator*(double2 a, double s) { return mk(a.x * s, a.y * s); }
__device__ __forceinline__ double2 cmul(double2 a, double2 b) { return mk(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
__device__ __forceinline__ double2 cmulc(double2 a, double2 b) { return mk(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y); }   // a conj(b)
__device__ __forceinline__ double2 mul_mi(double2 a) { return mk(a.y, -a.x); }   // -i a

// Register holding frequency m after dft<R>.
template <int R>
__host__ __device__ constexpr int reg_of(int m) {
    return R == 8 ? (m % 2 ? 4 + m / 2 : m / 2) : R == 9 ? 3 * (m % 3) + m / 3 : R == 16 ? 4 * (m % 4) + m / 4 : m;
}

// DFTs in registers, forward sign. 6, 10, 12, 15: two coprime factors
// (Good-Thomas, no twiddles); 8, 9, 16: two steps with twiddles, output left
// in register order (reg_of).
template <int R>
__device__ __forceinline__ void dft(double2 (&v)[R]) {
    if constexpr (R == 2) {
        const double2 a = v[0], b = v[1];
        v[0] = a + b;
        v[1] = a - b;
    } else if constexpr (R == 3) {
        constexpr double s = 0.866025403784438646763723170753;   // sin(2 pi / 3)
        const double2 t1 = v[1] + v[2], t2 = v[1] - v[2];
        const double2 a = mk(fma(-.5, t1.x, v[0].x), fma(-.5, t1.y, v[0].y));
        const double2 b = mul_mi(t2) * s;
        v[0] = v[0] + t1;
        v[1] = a + b;
        v[2] = a - b;
    } else if constexpr (R == 4) {
        const double2 a0 = v[0] + v[2], a1 = v[0] - v[2], a2 = v[1] + v[3], a3 = mul_mi(v[1] - v[3]);
        v[0] = a0 + a2;
        v[2] = a0 - a2;
        v[1] = a1 + a3;
        v[3] = a1 - a3;
    } else if constexpr (R == 5) {
        constexpr double c1 = 0.309016994374947424102293417183, s1 = 0.951056516295153572116439333379;   // cos, sin 2 pi / 5
        constexpr double c2 = -0.809016994374947424102293417183, s2 = 0.587785252292473129168705954639;  // ... 4 pi / 5
        const double2 t1 = v[1] + v[4], t2 = v[2] + v[3], t3 = v[1] - v[4], t4 = v[2] - v[3];
        const double2 a1 = v[0] + t1 * c1 + t2 * c2, a2 = v[0] + t1 * c2 + t2 * c1;
        const double2 b1 = mul_mi(t3 * s1 + t4 * s2), b2 = mul_mi(t3 * s2 - t4 * s1);
        v[0] = v[0] + t1 + t2;
        v[1] = a1 + b1;
        v[4] = a1 - b1;
        v[2] = a2 + b2;
        v[3] = a2 - b2;
    } else if constexpr (R == 8) {
        constexpr double h = 0.707106781186547524400844362105;
        double2 a[4], b[4], d[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            a[j] = v[j] + v[j + 4];
            d[j] = v[j] - v[j + 4];
        }
        b[0] = d[0];
        b[1] = mk(h * (d[1].x + d[1].y), h * (d[1].y - d[1].x));
        b[2] = mul_mi(d[2]);
        b[3] = mk(h * (d[3].y - d[3].x), -h * (d[3].x + d[3].y));
        dft<4>(a);
        dft<4>(b);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            v[j] = a[j];
            v[j + 4] = b[j];
        }
    } else if constexpr (R == 9) {
        // W9^1, W9^2, W9^4 = exp(-2 pi i k / 9)
        const double2 w1 = mk(0.766044443118978035202392650555, -0.642787609686539326322643409907);
        const double2 w2 = mk(0.173648177666930348851716626769, -0.984807753012208059366743024589);
        const double2 w4 = mk(-0.939692620785908384054109277325, -0.342020143325668733044099614682);
#pragma unroll
        for (int n2 = 0; n2 < 3; ++n2) {
            double2 a[3] = {v[n2], v[3 + n2], v[6 + n2]};
            dft<3>(a);
            v[n2] = a[0];
            v[3 + n2] = n2 == 0 ? a[1] : cmul(a[1], n2 == 1 ? w1 : w2);
            v[6 + n2] = n2 == 0 ? a[2] : cmul(a[2], n2 == 1 ? w2 : w4);
        }
#pragma unroll
        for (int k1 = 0; k1 < 3; ++k1) {
            double2 a[3] = {v[3 * k1], v[3 * k1 + 1], v[3 * k1 + 2]};
            dft<3>(a);
            v[3 * k1] = a[0];
            v[3 * k1 + 1] = a[1];
            v[3 * k1 + 2] = a[2];
        }
    } else if constexpr (R == 16) {
        constexpr double c = 0.923879532511286756128183189397, s = 0.382683432365089771728459984030;   // cos, sin pi / 8
        constexpr double h = 0.707106781186547524400844362105;
#pragma unroll
        for (int n2 = 0; n2 < 4; ++n2) {
            double2 a[4] = {v[n2], v[4 + n2], v[8 + n2], v[12 + n2]};
            dft<4>(a);
            // times W16^(n2 k1)
            v[n2] = a[0];
            if (n2 == 0) {
                v[4] = a[1];
                v[8] = a[2];
                v[12] = a[3];
            } else if (n2 == 1) {
                v[5] = cmul(a[1], mk(c, -s));
                v[9] = mk(h * (a[2].x + a[2].y), h * (a[2].y - a[2].x));
                v[13] = cmul(a[3], mk(s, -c));
            } else if (n2 == 2) {
                v[6] = mk(h * (a[1].x + a[1].y), h * (a[1].y - a[1].x));
                v[10] = mul_mi(a[2]);
                v[14] = mk(h * (a[3].y - a[3].x), -h * (a[3].x + a[3].y));
            } else {
                v[7] = cmul(a[1], mk(s, -c));
                v[11] = mk(h * (a[2].y - a[2].x), -h * (a[2].x + a[2].y));
                v[15] = cmul(a[3], mk(-c, s));
            }
        }
#pragma unroll
        for (int k1 = 0; k1 < 4; ++k1) {
            double2 a[4] = {v[4 * k1], v[4 * k1 + 1], v[4 * k1 + 2], v[4 * k1 + 3]};
            dft<4>(a);
#pragma unroll
            for (int k2 = 0; k2 < 4; ++k2) v[4 * k1 + k2] = a[k2];
        }
    } else {
        static_assert(R == 6 || R == 10 || R == 12, "radix");
        constexpr int A = R == 10 ? 2 : R == 6 ? 2 : 3, B = R / A;   // coprime
        // n = B n1 + A n2; frequency k with k = k1 mod A, k = k2 mod B
        double2 t[R];
#pragma unroll
        for (int n1 = 0; n1 < A; ++n1) {
            double2 b[B];
#pragma unroll
            for (int n2 = 0; n2 < B; ++n2) b[n2] = v[(B * n1 + A * n2) % R];
            dft<B>(b);
#pragma unroll
            for (int k2 = 0; k2 < B; ++k2) t[n1 * B + k2] = b[k2];
        }
        constexpr int ia = R == 12 ? 4 : R == 10 ? 5 : 3;    // = 1 mod A, 0 mod B
        constexpr int ib = R == 12 ? 9 : R == 10 ? 6 : 4;    // = 0 mod A, 1 mod B
#pragma unroll
        for (int k2 = 0; k2 < B; ++k2) {
            double2 a[A];
#pragma unroll
            for (int n1 = 0; n1 < A; ++n1) a[n1] = t[n1 * B + k2];
            dft<A>(a);
#pragma unroll
            for (int k1 = 0; k1 < A; ++k1) v[(ia * k1 + ib * k2) % R] = a[k1];
        }
    }
}

// fn(m, w^m) for m = 1 .. K: products at most four roundings deep, few live
// at a time.
template <int K, typename Fn>
__device__ __forceinline__ void powers(double2 w, const Fn& fn) {
    if constexpr (K <= 5) {
        double2 p[K + 1];
        p[1] = w;
        fn(1, w);
#pragma unroll
        for (int m = 2; m <= K; ++m) {
            p[m] = cmul(p[m / 2], p[m - m / 2]);
            fn(m, p[m]);
        }
    } else {
        const double2 w2 = cmul(w, w), w3 = cmul(w2, w), w4 = cmul(w2, w2);
        fn(1, w);
        fn(2, w2);
        fn(3, w3);
        double2 base = w4;
#pragma unroll
        for (int m = 4; m <= K; m += 4) {
            fn(m, base);
            if (m + 1 <= K) fn(m + 1, cmul(base, w));
            if (m + 2 <= K) fn(m + 2, cmul(base, w2));
            if (m + 3 <= K) fn(m + 3, cmul(base, w3));
            if (m + 4 <= K) base = m == 4 ? cmul(w4, w4) : cmul(base, w4);
        }
    }
}

// a / b and a % b, 0 <= a < 2^16: (a + 0.5) / b lies at least 0.5 / b from
// an integer, more than the float rounding.
__device__ __forceinline__ int div_small(int a, float inv) { return __float2int_rz(((float)a + 0.5f) * inv); }

// The CTA's F = 2^LF pairs in shared memory: element (position, pair f) at
// position * (F + 1) + f. The pitch is odd, so lanes along consecutive columns
// (positions an odd distance apart) and lanes along the pairs (F = 4: of two
// positions four apart, task_of) hit distinct banks, and the addresses of a butterfly
// stay linear.
template <int LF>
struct Shared {
    static_assert(LF == 2 || LF == 3, "4 or 8 pairs");
    static constexpr int F = 1 << LF, PITCH = F + 1;
    double2* S;
    __device__ __forceinline__ double2* at(int pos, int f) const { return S + pos * PITCH + f; }
    // task x of a pass whose lanes run over the pairs first: its position index
    static __device__ __forceinline__ int task_of(int x) {
        return LF == 3 ? x : (x & ~7) | (x & 1) << 2 | ((x >> 1) & 3);
    }
    static __device__ __forceinline__ int tasks(int count) { return LF == 3 ? count : (count + 7) & ~7; }
};

// d with its sign flipped where `mask` has the top bit set.
__device__ __forceinline__ double flip(double d, unsigned mask) {
    return __hiloint2double(__double2hiint(d) ^ (int)mask, __double2loint(d));
}

// First pass on the way forth. load(f, j, v): v[r] = element j + r M1 for
// r < R1/2, the mirrored (and, antisymmetric, negated) element
// (R1 - r) M1 - j for the others.
template <int R1, int LF, typename Load>
__device__ __forceinline__ void first_pass(const Shared<LF>& S, const F64Plan& p, const double2* tw, int type, const Load& load) {
    const float inv_ncol = 1.0f / (float)p.ncol, inv_rl = 1.0f / (float)p.RL;
    const int per = p.M1 / p.RL, step = per * S.PITCH;
    const unsigned neg = type ? 0x80000000u : 0u;
    for (int t = threadIdx.x; t < (p.ncol << LF); t += blockDim.x) {
        const int f = div_small(t, inv_ncol), j = t - f * p.ncol;
        const double2 w = __ldg(tw + j);
        double2 v[R1];
        load(f, j, v);
        if (type && j == 0) v[0] = v[R1 / 2] = mk(0.0, 0.0);
        dft<R1>(v);
        const int j2 = p.M1 - j;
        const int b0 = div_small(j, inv_rl), q0 = j - b0 * p.RL;
        const int b1 = div_small(j2, inv_rl), q1 = j2 - b1 * p.RL;
        double2* s0 = S.at(q0 * p.PB + b0, f);
        // columns 0 and M1 / 2 are their own mirrors: the second store goes
        // to the same place first, and the first one overwrites it
        double2* s1 = j > 0 ? S.at(q1 * p.PB + b1, f) : s0;
        const double2 v0 = v[reg_of<R1>(0)];
        s1[0] = mk(flip(v0.x, neg), flip(v0.y, neg));
        s0[0] = v0;
        powers<R1 / 2>(w, [&](int m, double2 wm) {
            const double2 y = cmulc(v[reg_of<R1>(m == R1 / 2 ? m : R1 - m)], wm);
            s1[m * step] = mk(flip(y.x, neg), flip(y.y, neg));
            s0[m * step] = cmul(v[reg_of<R1>(m)], wm);
        });
    }
}

// Last pass on the way back: store(f, j, v), v[reg_of(s)] the transform at
// j + s M1 (s < R1/2) or at the mirror (R1 - s) M1 - j (the others);
// ahead(f, j) comes before the task's shared-memory reads.
// ROWS_FAST: lanes along the columns (rows are written), else along the pairs
// (a transposed line is written).
template <int R1, bool ROWS_FAST, int LF, typename Ahead, typename Store>
__device__ __forceinline__ void last_pass(const Shared<LF>& S, const F64Plan& p, const double2* tw, int type, const Ahead& ahead,
                                          const Store& store) {
    const float inv_ncol = 1.0f / (float)p.ncol, inv_rl = 1.0f / (float)p.RL;
    const int per = p.M1 / p.RL, step = per * S.PITCH;
    const unsigned neg = type ? 0x80000000u : 0u;
    const int count = ROWS_FAST ? p.ncol << LF : S.tasks(p.ncol) << LF;
    for (int t = threadIdx.x; t < count; t += blockDim.x) {
        int f, j;
        if (ROWS_FAST) {
            f = div_small(t, inv_ncol);
            j = t - f * p.ncol;
        } else {
            f = t & (S.F - 1);
            j = S.task_of(t >> LF);
            if (LF < 3 && j >= p.ncol) continue;
        }
        const int j2 = j ? p.M1 - j : 0;
        const int b0 = div_small(j, inv_rl), q0 = j - b0 * p.RL;
        const int b1 = div_small(j2, inv_rl), q1 = j2 - b1 * p.RL;
        const double2 *s0 = S.at(q0 * p.PB + b0, f), *s1 = S.at(q1 * p.PB + b1, f);
        const double2 w = __ldg(tw + j);
        ahead(f, j);
        double2 v[R1];
        v[0] = s0[0];
        powers<R1 / 2>(w, [&](int m, double2 wm) {
            v[m] = cmul(s0[m * step], wm);
            if (m < R1 / 2) {
                const double2 y = cmulc(s1[m * step], wm);
                v[R1 - m] = mk(flip(y.x, neg), flip(y.y, neg));
            }
        });
        dft<R1>(v);
        store(f, j, v);
    }
}

// A middle radix on the way forth (BACK = false: DFT, then twiddles) or back
// (twiddles, then DFT), in place; `st`: product of the middle radices after it.
template <int R, bool BACK, int LF>
__device__ __forceinline__ void mid_pass(const Shared<LF>& S, const F64Plan& p, const double2* tw, int st) {
    const int nb = p.NB / R, count = nb * p.RL;
    const float inv_nb = 1.0f / (float)nb, inv_st = 1.0f / (float)st;
    const int tstep = p.P / (R * st * p.RL), step = st * S.PITCH;
    for (int t = threadIdx.x; t < (S.tasks(count) << LF); t += blockDim.x) {
        const int f = t & (S.F - 1), u = S.task_of(t >> LF);
        if (LF < 3 && u >= count) continue;
        const int q = div_small(u, inv_nb), e = u - q * nb;
        const int hi = div_small(e, inv_st), lo = e - hi * st;
        double2* s = S.at(q * p.PB + hi * R * st + lo, f);
        const double2 w = __ldg(tw + (lo * p.RL + q) * tstep);
        double2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = s[r * step];
        if constexpr (BACK) {
            powers<R - 1>(w, [&](int m, double2 wm) { v[m] = cmul(v[m], wm); });
            dft<R>(v);
#pragma unroll
            for (int r = 0; r < R; ++r) s[r * step] = v[reg_of<R>(r)];
        } else {
            dft<R>(v);
            s[0] = v[reg_of<R>(0)];
            powers<R - 1>(w, [&](int m, double2 wm) { s[m * step] = cmul(v[reg_of<R>(m)], wm); });
        }
    }
}

template <bool BACK, int LF>
__device__ __forceinline__ void mid_switch(int R, const Shared<LF>& S, const F64Plan& p, const double2* tw, int st) {
    switch (R) {
        case 2: mid_pass<2, BACK>(S, p, tw, st); break;
        case 3: mid_pass<3, BACK>(S, p, tw, st); break;
        case 4: mid_pass<4, BACK>(S, p, tw, st); break;
        case 5: mid_pass<5, BACK>(S, p, tw, st); break;
        case 6: mid_pass<6, BACK>(S, p, tw, st); break;
        case 8: mid_pass<8, BACK>(S, p, tw, st); break;
        case 9: mid_pass<9, BACK>(S, p, tw, st); break;
        case 10: mid_pass<10, BACK>(S, p, tw, st); break;
        case 12: mid_pass<12, BACK>(S, p, tw, st); break;
        default: mid_pass<16, BACK>(S, p, tw, st); break;
    }
}

template <int LF>
__device__ __forceinline__ void mids_forth(const Shared<LF>& S, const F64Plan& p, const double2* tw) {
    int st = p.NB / p.nsub;
    for (int i = 0; i < p.nmid; ++i) {
        st /= p.rm[i];
        mid_switch<false>(p.rm[i], S, p, tw, st);
        __syncthreads();
    }
}

template <int LF>
__device__ __forceinline__ void mids_back(const Shared<LF>& S, const F64Plan& p, const double2* tw) {
    int st = 1;
    for (int i = p.nmid - 1; i >= 0; --i) {
        mid_switch<true>(p.rm[i], S, p, tw, st);
        st *= p.rm[i];
        __syncthreads();
    }
}

#define F64_R1_SWITCH(R, call)            \
    switch (R) {                          \
        case 4: call(4); break;           \
        case 6: call(6); break;           \
        case 8: call(8); break;           \
        case 10: call(10); break;         \
        case 12: call(12); break;         \
        default: call(16); break;         \
    }
#define F64_RL_SWITCH(R, call)            \
    switch (R) {                          \
        case 2: call(2); break;           \
        case 3: call(3); break;           \
        case 4: call(4); break;           \
        case 5: call(5); break;           \
        case 6: call(6); break;           \
        case 8: call(8); break;           \
        case 9: call(9); break;           \
        default: call(10); break;         \
    }

__device__ __forceinline__ const F64Field& field_of(const F64Batch& b, int cta) {
    int fi = 0;
#pragma unroll 1
    for (int q = 1; q < b.count; ++q)
        if (cta >= b.f[q].cta_start) fi = q;
    return b.f[fi];
}

// First pass of A and B: pairs of rows of `in`, column c the transform's
// element c (0 .. L). Rows past the end repeat the last one (what comes of
// them goes to columns nobody reads). The first grid row of an antisymmetric
// axis 0 is not read either, the second stands in for it: its values are no part
// of the field, and as one of a pair they would reach the other row. ROTATE (A, which is not transformed
// back): an antisymmetric pair is read as i z, so that its transform is
// (X_a, X_b) as it stands; B leaves the factors of i and -1 to Lambda.
template <int R1, bool ROTATE, int LF>
__device__ __forceinline__ void load_rows(const Shared<LF>& S, const F64Plan& p, const double2* tw, const F64Field& F, int row0) {
    first_pass<R1>(S, p, tw, F.type, [&](int f, int j, double2 (&v)[R1]) {
        const int ra = max(min(row0 + 2 * f, F.rows - 1), F.border), rb = min(row0 + 2 * f + 1, F.rows - 1);
        const bool rot = ROTATE && F.type;
        const double* x = F.in + (ptrdiff_t)(rot ? rb : ra) * F.ld_in;
        const double* y = F.in + (ptrdiff_t)(rot ? ra : rb) * F.ld_in;
#pragma unroll
        for (int r = 0; r < R1; ++r) {
            const int c = r < R1 / 2 ? j + r * p.M1 : (R1 - r) * p.M1 - j;
            v[r] = mk(x[c], y[c]);
        }
        const unsigned fx = rot ? 0x80000000u : 0u, neg = F.type ? 0x80000000u : 0u;
#pragma unroll
        for (int r = 0; r < R1; ++r) {
            if (ROTATE) v[r].x = flip(v[r].x, r < R1 / 2 ? fx : 0u);   // i z = (-b, a), mirrored (b, -a)
            if (r >= R1 / 2) {
                if (!ROTATE) v[r].x = flip(v[r].x, neg);
                v[r].y = flip(v[r].y, neg);
            }
        }
    });
}

// A: rows along axis 1, out[p][grid row].
template <int LF>
__global__ void __launch_bounds__(F64_THREADS) fft64_a_kernel(const __grid_constant__ F64Batch b) {
    extern __shared__ __align__(16) unsigned char fft64_smem[];
    const F64Plan& p = b.p;
    const Shared<LF> S{reinterpret_cast<double2*>(fft64_smem)};
    const F64Field& F = field_of(b, blockIdx.x);
    const int row0 = (blockIdx.x - F.cta_start) * (2 << LF);
    pdl_wait();
#define CALL(R) load_rows<R, true>(S, p, b.tw, F, row0)
    F64_R1_SWITCH(p.R1, CALL)
#undef CALL
    __syncthreads();
    mids_forth(S, p, b.tw);
    auto last = [&](auto RC) {
        constexpr int R = decltype(RC)::value;
        for (int t = threadIdx.x; t < (S.tasks(p.NB) << LF); t += blockDim.x) {
            const int f = t & (S.F - 1), e = S.task_of(t >> LF);
            if (LF < 3 && e >= p.NB) continue;
            int to[R];
#pragma unroll
            for (int q = 0; q < R; ++q) to[q] = __ldg(F.tab + q * p.NB + e);
            const double2* s = S.at(e, f);
            const int step = p.PB * S.PITCH;
            double2 v[R];
#pragma unroll
            for (int q = 0; q < R; ++q) v[q] = s[q * step];
            dft<R>(v);
            double* o = F.out + row0 + 2 * f;
#pragma unroll
            for (int q = 0; q < R; ++q)
                if (to[q] >= 0) *reinterpret_cast<double2*>(o + to[q] * F.ld_out) = v[reg_of<R>(q)];
        }
    };
#define CALL(R) last(std::integral_constant<int, R>())
    F64_RL_SWITCH(p.RL, CALL)
#undef CALL
}

// B: rows along axis 0: forth, times Lambda, back; out[grid row][p].
template <int LF>
__global__ void __launch_bounds__(F64_THREADS) fft64_b_kernel(const __grid_constant__ F64Batch b) {
    extern __shared__ __align__(16) unsigned char fft64_smem[];
    __shared__ double red[F64_THREADS / 32];
    const F64Plan& p = b.p;
    const Shared<LF> S{reinterpret_cast<double2*>(fft64_smem)};
    const F64Field& F = field_of(b, blockIdx.x);
    const int row0 = (blockIdx.x - F.cta_start) * (2 << LF);
    pdl_wait();
#define CALL(R) load_rows<R, false>(S, p, b.tw, F, row0)
    F64_R1_SWITCH(p.R1, CALL)
#undef CALL
    __syncthreads();
    mids_forth(S, p, b.tw);
    // the last radix forth, Lambda, the same radix back. Antisymmetric rows:
    // Z = -i (X_a + i X_b) = (X_b, -X_a), and two factors of -i make -1, so
    // their Lambda pairs are stored swapped and negated.
    auto middle = [&](auto RC) {
        constexpr int R = decltype(RC)::value;
        for (int t = threadIdx.x; t < (S.tasks(p.NB) << LF); t += blockDim.x) {
            const int f = t & (S.F - 1), e = S.task_of(t >> LF);
            if (LF < 3 && e >= p.NB) continue;
            const double* l = F.lam + (ptrdiff_t)e * F.ld_lam + row0 + 2 * f;
            const int lstep = p.NB * F.ld_lam;
            double2 la[R];
#pragma unroll
            for (int q = 0; q < R; ++q) la[q] = __ldg(reinterpret_cast<const double2*>(l + q * lstep));
            double2* s = S.at(e, f);
            const int step = p.PB * S.PITCH;
            double2 v[R], g[R];
#pragma unroll
            for (int q = 0; q < R; ++q) v[q] = s[q * step];
            dft<R>(v);
#pragma unroll
            for (int q = 0; q < R; ++q) g[q] = mk(la[q].x * v[reg_of<R>(q)].x, la[q].y * v[reg_of<R>(q)].y);
            dft<R>(g);
#pragma unroll
            for (int q = 0; q < R; ++q) s[q * step] = g[reg_of<R>(q)];
        }
    };
#define CALL(R) middle(std::integral_constant<int, R>())
    F64_RL_SWITCH(p.RL, CALL)
#undef CALL
    __syncthreads();
    mids_back(S, p, b.tw);
    double psum = 0.0;
    auto store = [&](auto RC) {
        constexpr int R1 = decltype(RC)::value;
        last_pass<R1, false>(S, p, b.tw, F.type, [](int, int) {}, [&](int f, int j, double2 (&v)[R1]) {
            // a mirror written twice (columns 0 and M1 / 2) is written by one
            // thread, so which value stays does not vary
            double* o = F.out + row0 + 2 * f;
            const unsigned neg = F.type ? 0x80000000u : 0u;
#pragma unroll
            for (int s = 0; s < R1; ++s) {
                const int n = s < R1 / 2 ? j + s * p.M1 : (R1 - s) * p.M1 - j;
                double2 x = v[reg_of<R1>(s)];
                if (s >= R1 / 2) x = mk(flip(x.x, neg), flip(x.y, neg));
                *reinterpret_cast<double2*>(o + n * F.ld_out) = x;
            }
            if (F.sumw) {   // Bz (uniform per CTA)
                const double2 w = mk(F.sumw[row0 + 2 * f], F.sumw[row0 + 2 * f + 1]);
                const bool interior = j > 0 && 2 * j != p.M1;
                double2 x = mk(0.0, 0.0);
#pragma unroll
                for (int s = 0; s < R1; ++s)
                    if (s < R1 / 2 || interior || (s == R1 / 2 && j == 0)) x = x + v[reg_of<R1>(s)];
                psum += w.x * x.x + w.y * x.y;
            }
        });
    };
#define CALL(R) store(std::integral_constant<int, R>())
    F64_R1_SWITCH(p.R1, CALL)
#undef CALL
    if (F.partial) {   // uniform per CTA: fixed-order sum
#pragma unroll
        for (int o = 16; o; o >>= 1) psum += __shfl_xor_sync(0xffffffffu, psum, o);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = psum;
        __syncthreads();
        if (threadIdx.x == 0) {
            double s = 0.0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
            F.partial[blockIdx.x - F.cta_start] = s;
        }
    }
}

// Grid row of logical row r of D, or -1: rows whose transform is zero (the
// border, where axis 0 is antisymmetric) come last, as a pair of their own.
__device__ __forceinline__ int d_row(int r, int N, int border) {
    if (!border) return r < N ? r : -1;
    return r < N - 2 ? r + 1 : r == N - 1 ? 0 : r == N ? N - 1 : -1;
}

// D: rows along axis 1, back only; the field itself, finalised.
template <int LF>
__global__ void __launch_bounds__(F64_THREADS) fft64_d_kernel(const __grid_constant__ F64Batch b) {
    extern __shared__ __align__(16) unsigned char fft64_smem[];
    __shared__ double s_mean;
    const F64Plan& p = b.p;
    const Shared<LF> S{reinterpret_cast<double2*>(fft64_smem)};
    const F64Field& F = field_of(b, blockIdx.x);
    const int row0 = (blockIdx.x - F.cta_start) * (2 << LF);   // logical row
    pdl_wait();
    if (F.partial && threadIdx.x < 32) {   // the sum over the grid, in a fixed order
        double s = 0.0;
        for (int k = threadIdx.x; k < F.npartial; k += 32) s += F.partial[k];
#pragma unroll
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (threadIdx.x == 0) s_mean = s * F.inv_n;
    }
    auto first = [&](auto RC) {
        constexpr int R = decltype(RC)::value;
        const float inv_nb = 1.0f / (float)p.NB;
        for (int t = threadIdx.x; t < (p.NB << LF); t += blockDim.x) {
            const int f = div_small(t, inv_nb), e = t - f * p.NB;
            int c[R];
#pragma unroll
            for (int q = 0; q < R; ++q) c[q] = __ldg(F.tab + q * p.NB + e);
            const int r = row0 + 2 * f;
            const int ga = d_row(r, p.N, F.border), gb = d_row(r + 1, p.N, F.border);
            // a pair of border rows, and the pairs past the end, read zeros
            // (column `zero`); a last single row is paired with itself
            const bool none = r >= p.N - 2 * F.border;
            const double* ra = F.in + (ptrdiff_t)max(ga, 0) * F.ld_in;
            const double* rb = F.in + (ptrdiff_t)max(gb, 0) * F.ld_in;
            if (!none && gb < 0) rb = ra;
            // antisymmetric: read as i z, so the transform is (F_a, F_b)
            const double* x = F.type ? rb : ra;
            const double* y = F.type ? ra : rb;
            const unsigned fx = F.type ? 0x80000000u : 0u;
            double2 v[R];
#pragma unroll
            for (int q = 0; q < R; ++q) {
                const int cq = none ? F.zero : c[q] & 0x7fffffff;
                v[q] = mk(x[cq], y[cq]);
            }
#pragma unroll
            for (int q = 0; q < R; ++q) {
                const unsigned sg = (unsigned)c[q] & 0x80000000u;
                v[q] = mk(flip(v[q].x, sg ^ fx), flip(v[q].y, sg));
            }
            dft<R>(v);
            double2* s = S.at(e, f);
            const int step = p.PB * S.PITCH;
#pragma unroll
            for (int q = 0; q < R; ++q) s[q * step] = v[reg_of<R>(q)];
        }
    };
#define CALL(R) first(std::integral_constant<int, R>())
    F64_RL_SWITCH(p.RL, CALL)
#undef CALL
    __syncthreads();
    mids_back(S, p, b.tw);
    const double mean = F.partial ? s_mean : 0.0;
    auto store = [&](auto RC) {
        constexpr int R1 = decltype(RC)::value;
        // the previous field of the pair's first row is loaded before the
        // pass's shared-memory reads and butterfly, that of the second row as
        // the first one's values are stored
        double old[R1];
        auto row_of = [&](int f, int h) { return d_row(row0 + 2 * f + h, p.N, F.border); };
        auto n_of = [&](int j, int s) { return s < R1 / 2 ? j + s * p.M1 : (R1 - s) * p.M1 - j; };
        auto ahead = [&](int f, int j) {
            const int g = row_of(f, 0);
            if (F.avg && g >= 0) {
                const double* pr = F.prev + g * p.N;
#pragma unroll
                for (int s = 0; s < R1; ++s) old[s] = pr[n_of(j, s)];
            }
        };
        last_pass<R1, true>(S, p, b.tw, F.type, ahead, [&](int f, int j, double2 (&v)[R1]) {
            const unsigned neg = F.type ? 0x80000000u : 0u;
            const bool interior = j > 0 && 2 * j != p.M1;   // the other columns are their own mirrors
            if (F.type && j == 0) v[reg_of<R1>(0)] = v[reg_of<R1>(R1 / 2)] = mk(0.0, 0.0);
            const int gb = row_of(f, 1);
            const double* next = F.avg && gb >= 0 ? F.prev + gb * p.N : nullptr;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int g = h ? gb : row_of(f, 0);
                if (g < 0) continue;
                double* o = F.out ? F.out + g * p.N : nullptr;
                double* a = F.avg ? F.avg + g * p.N : nullptr;
#pragma unroll
                for (int s = 0; s < R1; ++s) {
                    const int n = n_of(j, s);
                    const double2 z = v[reg_of<R1>(s)];
                    double x = h ? z.y : z.x;
                    if (s >= R1 / 2) x = flip(x, neg);
                    x -= mean;
                    if (F.variant_a) x = 2 * x - old[s];
                    if (s < R1 / 2 || interior || (s == R1 / 2 && j == 0)) {
                        if (o) o[n] = x;
                        if (a) a[n] = (x + old[s]) / 2;
                    }
                    if (h == 0 && next) old[s] = next[n];
                }
            }
        });
    };
#define CALL(R) store(std::integral_constant<int, R>())
    F64_R1_SWITCH(p.R1, CALL)
#undef CALL
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

// Lambda in the order the passes have it in: out[t][p] = lam[k0 of t][k1 of p],
// 0 where the transform has no such frequency.
// swap: pairs of columns swapped and negated (antisymmetric rows, fft64_b_kernel).
__global__ void lam_order_kernel(const double* __restrict__ lam, int ld, const int* __restrict__ k0, int T,
                                 const int* __restrict__ k1, int cols, int swap, double* __restrict__ out, int ld_out) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x, t = blockIdx.y;
    if (c >= ld_out) return;
    const double v = c < cols && k0[t] >= 0 ? lam[(size_t)k0[t] * ld + k1[c]] : 0.0;
    out[(size_t)t * ld_out + (swap ? c ^ 1 : c)] = swap ? -v : v;
}

constexpr int F64_SMALL = 400, F64_MEDIUM = 1100;   // rows: see fft64_init

// The radices of P. One middle radix where there is such a plan: two passes
// need radices so large, and four so many barriers, that both are slower (us
// per xi step: 41^2 8 10 66.8, 4 5 4 63.8, 81^2 16 10 74.0, 8 5 4 67.9; 161^2
// 8 8 5 76.2, 4 5 4 4 79.1; 641^2 16 8 10 363.7, 16 4 5 4 377.0). Then the
// smallest sum of radices, the length of the chain a butterfly is; then the
// fewest kept positions; then, on large grids, the larger last radix (641^2
// 16 8 10 362, 16 10 8 368) and on small ones the smaller (161^2 8 8 5 76.2,
// 8 5 8 78.1), B's longest pass being its middle one.
bool make_plan(int N, F64Plan* out) {
    static const int first[] = {16, 12, 10, 8, 6, 4}, mid[] = {16, 12, 10, 9, 8, 6, 5, 4, 3, 2},
                     last[] = {10, 9, 8, 6, 5, 4, 3, 2};
    F64Plan p{}, best{};
    p.N = N;
    p.L = N - 1;
    p.P = 2 * p.L;
    long long best_cost = -1;
    auto consider = [&]() {
        long long sum = p.R1 + p.RL;
        for (int i = 0; i < p.nmid; ++i) sum += p.rm[i];
        const long long mids = p.nmid > 1 ? p.nmid - 1 : 1 - p.nmid;
        const long long cost = ((mids * 1000 + sum) * 100000 + (p.R1 / 2 + 1) * p.M1) * 32 + (N < F64_SMALL ? p.RL : 31 - p.RL);
        if (best_cost < 0 || cost < best_cost) {
            best_cost = cost;
            best = p;
        }
    };
    auto rec = [&](auto&& self, int rem) -> void {
        for (int r : last)
            if (r == rem) {
                p.RL = r;
                consider();
            }
        if (p.nmid >= MAX_MIDS) return;
        for (int r : mid)
            if (rem % r == 0 && rem / r > 1) {
                p.rm[p.nmid++] = r;
                self(self, rem / r);
                --p.nmid;
            }
    };
    for (int r : first)
        if (p.P % r == 0 && p.P / r > 1) {
            p.R1 = r;
            p.M1 = p.P / r;
            rec(rec, p.M1);
        }
    if (best_cost < 0) return false;
    best.nsub = best.R1 / 2 + 1;
    best.ncol = best.M1 / 2 + 1;
    best.NB = best.nsub * best.M1 / best.RL;
    best.PB = best.NB | 1;
    *out = best;
    return true;
}

size_t smem_bytes(const F64Plan& p) { return (size_t)p.RL * p.PB * ((1 << p.lf) + 1) * sizeof(double2); }

constexpr size_t F64_MAX_SMEM = 225 * 1024;

struct F64State {
    F64Plan p;
    int threads, T;
    int pitch;              // of the intermediates and Lambda
    int zero;               // a column of the intermediates that is never written
    int kept[2];            // kept frequencies of the two types
    int* tabs;              // device: A tables (2 T), D tables (2 T), k0 (2 T), k1 (2 pitch)
    double* lam[3 + 1];     // by type0 * 2 + type1
    double* sumw;
};

using F64Kernel = void (*)(F64Batch);
F64Kernel kernel_of(int pass, int lf) {
    static const F64Kernel k[3][2] = {{fft64_a_kernel<2>, fft64_a_kernel<3>},
                                      {fft64_b_kernel<2>, fft64_b_kernel<3>},
                                      {fft64_d_kernel<2>, fft64_d_kernel<3>}};
    return k[pass][lf - 2];
}

const int* tab_a(const F64State* s, int type) { return s->tabs + type * s->T; }
const int* tab_d(const F64State* s, int type) { return s->tabs + (2 + type) * s->T; }

}  // namespace

// Row pitch of the intermediates: the rows of whole CTAs, then a column of
// zeros (the planes are cleared once, at set-up).
int fft64_pitch(int N) { return (N + 15) / 16 * 16 + 16; }

int fft64_init(lc3d_ctx* c) {
    F64Plan p{};
    if (!make_plan(c->N, &p)) return LC3D_ERR_PARAM;
    const int N = c->N, L = p.L;
    F64State* s = new F64State();
    c->fft64 = s;
    // Pairs and threads per CTA: 256 threads and two CTAs per SM where the
    // shared memory allows, else 512 threads and one. Eight pairs store whole
    // lines and fill the SMs from about 400 rows on; smaller grids take four,
    // for twice the CTAs, and so do those of 700 to 1100 rows, of which eight
    // pairs fit an SM once and four twice (us per xi step, F = 8 / F = 4, around
    // the lines: 321^2 129.0 / 119.4, 401^2 199 / 222; 641^2 372 / 430, 801^2
    // 621 / 600; 1025^2 927 / 913, 1153^2 1118 / 1156).
    auto twice = [&](int lf) {
        p.lf = lf;
        return 2 * (smem_bytes(p) + 2048) <= 228 * 1024;
    };
    int lf = 3;
    if (N < F64_SMALL || (N <= F64_MEDIUM && !twice(3) && twice(2))) lf = 2;
    s->threads = twice(lf) ? 256 : 512;
    if (smem_bytes(p) > F64_MAX_SMEM) p.lf = 2;
    if (smem_bytes(p) > F64_MAX_SMEM) return LC3D_ERR_SIZE;
    s->p = p;
    s->pitch = fft64_pitch(N);
    s->zero = s->pitch - 1;
    const int T = s->T = p.RL * p.NB;
    // frequency of every position (butterfly b, element q of the last radix)
    std::vector<int> freq(T);
    for (int q = 0; q < p.RL; ++q)
        for (int b = 0; b < p.NB; ++b) {
            int per = p.NB / p.nsub, rest = b % per, k = b / per, mul = p.R1;
            for (int i = 0; i < p.nmid; ++i) {
                per /= p.rm[i];
                k += mul * (rest / per);
                rest %= per;
                mul *= p.rm[i];
            }
            freq[q * p.NB + b] = k + mul * q;
        }
    std::vector<int> tabs(6 * T + 2 * s->pitch, 0);
    for (int type = 0; type < 2; ++type) {
        int* ta = tabs.data() + type * T;
        int* td = tabs.data() + (2 + type) * T;
        int* k0 = tabs.data() + (4 + type) * T;
        int* k1 = tabs.data() + 6 * T + type * s->pitch;
        std::vector<int> col(p.P, -1);   // of a kept extended frequency
        int n = 0;
        for (int t = 0; t < T; ++t) {
            const int k = freq[t], m = k % p.R1, kk = k <= L ? k : p.P - k;
            const bool zero = type && (kk == 0 || kk == L);
            const bool dup = k > L && (m == 0 || m == p.R1 / 2);   // its mirror is kept
            k0[t] = zero ? -1 : kk - type;
            ta[t] = zero || dup ? -1 : n;
            if (ta[t] >= 0) {
                col[k] = n;
                k1[n++] = kk - type;
            }
        }
        s->kept[type] = n;
        for (int t = 0; t < T; ++t) {
            const int k = freq[t];
            if (k0[t] < 0) td[t] = s->zero;
            else if (ta[t] >= 0) td[t] = ta[t];
            else td[t] = (int)((unsigned)col[p.P - k] | (type ? 0x80000000u : 0u));
        }
        if (n != N - 2 * type) return LC3D_ERR_PARAM;
    }
    LC3D_CUDA_TRY(cudaMalloc(&s->tabs, tabs.size() * sizeof(int)));
    LC3D_CUDA_TRY(cudaMemcpy(s->tabs, tabs.data(), tabs.size() * sizeof(int), cudaMemcpyHostToDevice));
    // the sum over grid columns of cos(pi k j / L), j = 0 .. L, is N at k = 0,
    // 1 at other even k and 0 at odd k; k and P - k count for one kept k
    std::vector<double> w(s->pitch + 16, 0.0);
    for (int n = 0; n < s->kept[0]; ++n) {
        const int k = tabs[6 * T + n];
        w[n] = k == 0 ? (double)N : k % 2 ? 0.0 : k == L ? 1.0 : 2.0;
    }
    LC3D_CUDA_TRY(cudaMalloc(&s->sumw, w.size() * sizeof(double)));
    LC3D_CUDA_TRY(cudaMemcpy(s->sumw, w.data(), w.size() * sizeof(double), cudaMemcpyHostToDevice));
    const double* src[4] = {c->lam_neu, c->lam_mixT, c->lam_mix, c->lam_dir};
    for (int k = 0; k < 4; ++k) {
        const int type0 = k >> 1, type1 = k & 1, cols = N - 2 * type1;
        LC3D_CUDA_TRY(cudaMalloc(&s->lam[k], (size_t)T * s->pitch * sizeof(double)));
        lam_order_kernel<<<dim3((s->pitch + 127) / 128, T), 128>>>(src[k], cols, s->tabs + (4 + type0) * T, T,
                                                                    s->tabs + 6 * T + type1 * s->pitch, cols, type0,
                                                                    s->lam[k], s->pitch);
        LC3D_CUDA_TRY(cudaGetLastError());
    }
    fields_drop_lam(c);   // this state has its own, in its order
    for (int pass = 0; pass < 3; ++pass)   // per kernel, not per context: the largest any context may use
        LC3D_CUDA_TRY(cudaFuncSetAttribute(kernel_of(pass, p.lf), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)F64_MAX_SMEM));
    return LC3D_OK;
}

void fft64_free(lc3d_ctx* c) {
    F64State* s = static_cast<F64State*>(c->fft64);
    if (!s) return;
    if (s->tabs) cudaFree(s->tabs);
    if (s->sumw) cudaFree(s->sumw);
    for (double* l : s->lam)
        if (l) cudaFree(l);
    delete s;
    c->fft64 = nullptr;
}

int fft64_solve(lc3d_ctx* c, const Fft64Desc* desc, int count, cudaStream_t s) {
    const F64State* st = static_cast<const F64State*>(c->fft64);
    const F64Plan& p = st->p;
    const int rows_cta = 2 << p.lf, N = c->N;
    const size_t smem = smem_bytes(p);
    for (int pass = 0; pass < 3; ++pass) {
        F64Batch b;
        memset(&b, 0, sizeof(b));
        b.p = p;
        b.tw = reinterpret_cast<const double2*>(c->fft_tw);
        b.count = count;
        int ctas = 0;
        for (int q = 0; q < count; ++q) {
            const Fft64Desc& d = desc[q];
            F64Field& f = b.f[q];
            const int n1 = N - 2 * d.type1;
            f.cta_start = ctas;
            f.ld_out = st->pitch;
            int rows = N;
            if (pass == 0) {        // all grid rows: what comes of an antisymmetric axis 0's border rows is read by nobody
                f.in = d.rhs; f.ld_in = N; f.rows = N; f.type = d.type1;
                f.out = d.t1;
                f.tab = tab_a(st, d.type1);
                f.border = d.type0;
            } else if (pass == 1) {
                f.in = d.t1; f.ld_in = st->pitch; f.rows = rows = n1; f.type = d.type0;
                f.out = d.t2;
                f.lam = st->lam[d.type0 * 2 + d.type1];
                f.ld_lam = st->pitch;
                if (d.sums) {
                    f.partial = d.sums;
                    f.sumw = st->sumw;
                }
            } else {
                f.in = d.t2; f.ld_in = st->pitch; f.type = d.type1;
                f.border = d.type0;
                f.zero = st->zero;
                rows = N + f.border;
                f.tab = tab_d(st, d.type1);
                f.out = d.out; f.avg = d.avg; f.prev = d.prev;
                f.variant_a = d.variant_a;
                if (d.sums) {
                    f.partial = d.sums;
                    f.npartial = (n1 + rows_cta - 1) / rows_cta;
                    f.inv_n = 1.0 / ((double)N * N);
                }
            }
            ctas += (rows + rows_cta - 1) / rows_cta;
        }
        if (!ctas) return LC3D_OK;
        ProfScope ps(c, LC3D_STAGE_TRANSFORM, s);
        LC3D_CUDA_TRY(launch_pdl(kernel_of(pass, p.lf), dim3(ctas), dim3(st->threads), smem, s, b));
        LC3D_CUDA_TRY(cudaGetLastError());
    }
    return LC3D_OK;
}
