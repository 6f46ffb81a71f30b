"""The deposition kernel's own source, compiled for the CPU and run with its
warps in either order: one fiber per thread, switched at the barriers only, so
the first warp runs either ahead of all others or behind them. CUDA orders the
warps of a CTA nowhere but at its barriers, so both have to give the density."""
import re
import subprocess

import numpy as np
import pytest

from conftest import ROOT, GOLDEN  # noqa: F401
from make_golden import make_config
from oracle import lcode_oracle as O

SHIM = r'''
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <ucontext.h>
#include <vector>
using std::min; using std::max;
#define __device__
#define __host__
#define __global__
#define __forceinline__ inline
#define __shared__ static
#define __align__(n) alignas(n)
struct double2 { double x, y; };
struct uint4 { unsigned x, y, z, w; };
static double2 make_double2(double x, double y) { return {x, y}; }
static uint4 make_uint4(unsigned x, unsigned y, unsigned z, unsigned w) { return {x, y, z, w}; }
struct Dim { int x; };
// fiber scheduler: state 0 runnable, 1 at a CTA barrier, 2 at a warp barrier, 3 done
static int g_threads, g_now, g_state[1024], g_red[1024];
static ucontext_t g_main, g_ctx[1024];
#define threadIdx (Dim{g_now})
static void wait_at(int state) {
    g_state[g_now] = state;
    swapcontext(&g_ctx[g_now], &g_main);
}
static void __syncthreads() { wait_at(1); }
static void __syncwarp() { wait_at(2); }
template <typename F> static int warp_reduce(int v, F f) {
    g_red[g_now] = v;
    wait_at(2);
    int r = v;
    for (int l = 0; l < 32; ++l) r = f(r, g_red[(g_now & ~31) + l]);
    wait_at(2);
    return r;
}
static int __reduce_min_sync(unsigned, int v) { return warp_reduce(v, [](int a, int b) { return min(a, b); }); }
static int __reduce_max_sync(unsigned, int v) { return warp_reduce(v, [](int a, int b) { return max(a, b); }); }
static void atomicMin(int* p, int v) { *p = min(*p, v); }
static void atomicMax(int* p, int v) { *p = max(*p, v); }
static void atomicOr(unsigned* p, unsigned v) { *p |= v; }
static void atomicAdd(unsigned long long* p, unsigned long long v) { *p += v; }
template <typename T> static T __ldg(const T* p) { return *p; }
static int __ffs(unsigned v) { return v ? __builtin_ctz(v) + 1 : 0; }
static int __float2int_rz(float v) { return (int)v; }
static int __double2loint(double d) { int64_t b; memcpy(&b, &d, 8); return (int)b; }
static long long __double_as_longlong(double d) { long long b; memcpy(&b, &d, 8); return b; }
static void pdl_wait() {}
#define LC3D_FLAG_WINDOW 0
#define LC3D_FLAG_NONFINITE 1
static void raise_flag(unsigned* err, int flag) { err[flag] = 1; }
'''

MAIN = r'''
static DepositArgs g_args;
static int g_tx, g_ty;
static void body() {
    deposit_tile<TI, RPW, FS>(g_args, g_tx, g_ty);
    g_state[g_now] = 3;
    swapcontext(&g_ctx[g_now], &g_main);
}
// One CTA; last_first: always run the runnable thread of the highest index, else of the lowest.
static void run_cta(std::vector<std::vector<char>>& stacks, bool last_first) {
    memset(smem_f64, 0xff, sizeof(smem_f64));
    for (int t = 0; t < g_threads; ++t) {
        getcontext(&g_ctx[t]);
        g_ctx[t].uc_stack.ss_sp = stacks[t].data();
        g_ctx[t].uc_stack.ss_size = stacks[t].size();
        g_ctx[t].uc_link = &g_main;
        makecontext(&g_ctx[t], body, 0);
        g_state[t] = 0;
    }
    for (;;) {
        int next = -1;
        for (int k = 0; k < g_threads && next < 0; ++k) {
            const int t = last_first ? g_threads - 1 - k : k;
            if (g_state[t] == 0) next = t;
        }
        if (next >= 0) {
            g_now = next;
            swapcontext(&g_main, &g_ctx[next]);
            // a whole warp at a warp barrier goes on
            const int w = next & ~31;
            bool all = true;
            for (int t = w; t < w + 32; ++t) all = all && g_state[t] == 2;
            for (int t = w; all && t < w + 32; ++t) g_state[t] = 0;
            continue;
        }
        int done = 0;
        for (int t = 0; t < g_threads; ++t) done += g_state[t] == 3;
        if (done == g_threads) return;
        for (int t = 0; t < g_threads; ++t) {
            if (g_state[t] == 2) { fprintf(stderr, "a warp barrier not every lane reaches\n"); exit(2); }
            if (g_state[t] == 1) g_state[t] = 0;
        }
    }
}
int main(int argc, char** argv) {
    FILE* f = fopen(argv[1], "rb");
    int n[4];
    double g[2];
    if (fread(n, 4, 4, f) != 4 || fread(g, 8, 2, f) != 2) return 1;
    const int Nc = n[0], Nf = n[1], N = n[2];
    auto doubles = [&](size_t k) { std::vector<double> v(k); if (fread(v.data(), 8, k, f) != k) exit(1); return v; };
    std::vector<std::vector<double>> c, l;
    for (int k = 0; k < 7; ++k) c.push_back(doubles((size_t)Nc * Nc));
    for (int k = 0; k < 3; ++k) l.push_back(doubles(Nf));
    std::vector<int32_t> ip(Nf), in(Nf);
    if (fread(ip.data(), 4, Nf, f) != (size_t)Nf || fread(in.data(), 4, Nf, f) != (size_t)Nf) return 1;
    fclose(f);
    g_threads = dep_threads(TI, RPW);
    std::vector<std::vector<char>> stacks(g_threads, std::vector<char>(65536));
    FILE* o = fopen(argv[2], "wb");
    for (int order = 0; order < 2; ++order) {
        std::vector<unsigned long long> acc((size_t)8 * N * N, 0);
        unsigned err[3] = {};
        DepositArgs& a = g_args;
        a = DepositArgs{};
        a.x_offt = c[0].data(); a.y_offt = c[1].data(); a.m = c[2].data(); a.q = c[3].data();
        a.px = c[4].data(); a.py = c[5].data(); a.pz = c[6].data();
        a.inf_prev = l[0].data(); a.inf_next = l[1].data(); a.fine_grid = l[2].data();
        a.idx_prev = ip.data(); a.idx_next = in.data();
        a.acc = acc.data(); a.plane = (size_t)N * N;
        a.Nc = Nc; a.Nf = Nf; a.N = N; a.fine_off = n[3];
        a.h = g[0]; a.inv_h = 1 / g[0]; a.sf = g[1];
        a.err = err;
        const int tx = (Nf + n[3] + DEP_TW - 1) / DEP_TW, ty = (Nf + n[3] + TI - 1) / TI;
        for (g_ty = 0; g_ty < ty; ++g_ty)
            for (g_tx = 0; g_tx < tx; ++g_tx) run_cta(stacks, order == 1);
        std::vector<double> out((size_t)4 * N * N);
        for (int q = 0; q < 4; ++q)
            for (int k = 0; k < N * N; ++k)
                out[(size_t)q * N * N + k] = (double)(long long)acc[(size_t)2 * q * N * N + k] * 0x1p-24 +
                                             (double)(long long)acc[(size_t)(2 * q + 1) * N * N + k] * 0x1p-76;
        fwrite(out.data(), 8, out.size(), o);
        fwrite(err, 4, 3, o);
    }
    fclose(o);
}
'''


def program(tmp_path, rows, per_warp, split):
    src = open(f'{ROOT}/lcode3d_b200/csrc/particles.cu').read()
    args = re.search(r'struct DepositArgs \{.*?\n\};\n', open(f'{ROOT}/lcode3d_b200/csrc/lc3d_internal.cuh').read(), re.S).group(0)
    body = src[src.index('struct Tsc {'):src.index('// Field-free estimate')]
    body += src[src.index('constexpr double FX_MAX'):src.index('// One tile per CTA')]
    # the hardware's approximations stand for a good first guess
    body = re.sub(r'asm\("rsqrt\.approx.*', 'y = 1 / std::sqrt(S);', body)
    body = re.sub(r'asm\("rcp\.approx.*', 'r = 1 / d;', body)
    body = re.sub(r'extern __shared__ .*\n', '', body)
    cpp = tmp_path / 'deposit.cpp'
    cpp.write_text(SHIM + 'alignas(16) static double smem_f64[29056];\n' + args + body + f'#define TI {rows}\n#define RPW {per_warp}\n#define FS {split}\n' + MAIN)
    exe = tmp_path / 'deposit'
    subprocess.run(['g++', '-O1', '-std=c++17', '-w', '-o', str(exe), str(cpp)], check=True)
    return exe


@pytest.mark.parametrize('rows, per_warp, split', [(12, 3, 1), (4, 3, 1), (4, 1, 1), (4, 1, 2), (4, 1, 4)])
def test_deposit_does_not_depend_on_the_order_of_warps(tmp_path, rows, per_warp, split):
    N, coarse, fine = 41, 3, 2
    cfg = make_config(N, 0.1, 0.05, 10, amplitude=0.3)
    x0, y0, *_, m, q, virt = O.make_plasma(N - 2 * cfg.plasma_padding_steps, 0.1, coarse, fine)
    rng = np.random.default_rng(3)
    x, y = (0.1 * np.sin(x0 + 2 * y0 + k) + 0.02 * rng.normal(size=x0.shape) for k in range(2))
    p = [0.3 * rng.normal(size=x0.shape) for _ in range(3)]
    coarse_arrays = [x, y, m, q, *p]
    want = O.deposit(cfg, 0, *coarse_arrays, virt)
    data = tmp_path / 'in'
    with open(data, 'wb') as f:
        np.array([x0.shape[0], len(virt.fine_grid), N, 1], dtype=np.int32).tofile(f)   # even fineness: offset 1
        np.array([0.1, 1 / (coarse * fine) ** 2]).tofile(f)
        for a in (*coarse_arrays, virt.influence_prev, virt.influence_next, virt.fine_grid):
            np.ascontiguousarray(a, dtype=np.float64).tofile(f)
        for a in (virt.indices_prev, virt.indices_next):
            np.ascontiguousarray(a, dtype=np.int32).tofile(f)
    out = tmp_path / 'out'
    subprocess.run([str(program(tmp_path, rows, per_warp, split)), str(data), str(out)], check=True, timeout=300)
    raw = out.read_bytes()
    size = 4 * N * N * 8 + 12
    orders = [np.frombuffer(raw[k * size:k * size + size - 12]).reshape(4, N, N) for k in range(2)]
    for order, got in zip(('first warp first', 'first warp last'), orders):
        for name, g, w in zip(('ro', 'jx', 'jy', 'jz'), got, want):
            assert O.relative_error(g, w) < 1e-13, (order, name)   # the particle stages' parity tolerance
    assert np.array_equal(*orders)
