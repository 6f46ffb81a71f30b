// Learned field predictor: a small convolutional U-Net that predicts the
// first-pass (predictor-stage) fields Ex, Ey, Bx, By, Bz of the next xi
// step from the fields of the two previous steps, so that the solver can
// skip the first deposit + field solve of lcode.py:846-871 (the pass that
// moves the particles with the previous step's fields, "no halfstep-averaged
// fields yet") and go straight to the corrector. No counterpart in the
// reference; the corrector that follows is the reference's own
// (lcode.py:882-911) and judges the prediction.
//
// Network (all 3x3 convolutions, BF16 weights and activations, FP32
// accumulation, sum skip connections):
//   x0  (27 of 32 channels)          N x N      normalised fields of t-1, t-1 minus t-2, levels
//   e1 = relu(conv1(x0))     32      N x N
//   e2 = relu(conv2(pool(e1))) 64    N2 x N2    N2 = (N + 1) / 2
//   e3 = relu(conv3(pool(e2))) 128   N3 x N3    N3 = (N2 + 1) / 2
//   u3 = conv4(e3)           64      N3 x N3
//   d2 = relu(up(u3) + e2)   64      N2 x N2    up: nearest neighbour
//   u2 = conv5(d2)           32      N2 x N2
//   d1 = relu(up(u2) + e1)   32      N x N
//   y  = conv6(d1)           16 (5 used), float32
// prediction = 2 F(t-1) - F(t-2) + out_scale * y (per field), i.e. the
// network learns the correction to linear extrapolation.
//
// Layout. An activation at a level with H x W pixels is [H][W + 1][C]
// (NHWC, row pitch Wp = W + 1): column W of every row is kept zero, so in
// the flattened pixel index p = y Wp + x the 3x3 neighbours of p are
// p + dy Wp + dx and the zero column doubles as the left/right padding;
// rows above and below fall outside [0, H Wp) and are zero-filled by TMA.
//
// Inference convolution: implicit GEMM on the 5th-generation tensor cores.
// A CTA owns 128 consecutive flattened pixels (M = 128) and all output
// channels (N = Cout); K runs over 9 taps x Cin in blocks of 32 channels.
// Per K block warp 0 TMA-loads the 128 x 32 input tile shifted by the tap
// (a 2-D tensor map over [H Wp][Cin], 64-byte swizzle) and the Cout x 32
// weight tile of that tap, warp 1 issues two tcgen05.mma (128 x Cout x 16,
// bf16 -> f32 in TMEM), warps 2-5 add the bias, apply ReLU and store bf16
// (or f32) NHWC, writing zeros in the pad column. Every mbarrier wait is
// bounded; on time-out the kernel sets an error flag and exits, and TMEM is
// always freed.
//
// Training: both gradient passes of every convolution on the tensor cores
// in bf16 -- the data gradient as the forward convolution of the bf16 output
// gradient with flipped, transposed weights, the weight gradient as an
// implicit GEMM over pixels with MN-major operands -- and SIMT kernels for an
// MSE loss on the 5 fields, the pooling / upsampling / ReLU adjoints, which
// write the output gradients in bf16 and sum the bias gradients on the way,
// and Adam. Weights are kept as float32 master
// copies; the bf16 copies the forward pass reads are refreshed after every
// update.

#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "lc3d.h"
#include "lc3d_internal.cuh"
#include "tc_sm100.cuh"

namespace {

using namespace tc;

constexpr int NLAYERS = 6;
constexpr int CONV_THREADS = 192;
constexpr int CONV_STAGES = 4;
constexpr int TILE_PIX = 128;                      // M
constexpr int KB = 32;                             // channels per K block (64 bytes of bf16)
constexpr int A_TILE_BYTES = TILE_PIX * KB * 2;     // 8 KiB

// Bytes of a pipeline stage's weight tile: Cout rows of 64 bytes, at least
// 1 KiB (the 64-byte swizzle's alignment); smaller layers take less shared
// memory, so more CTAs are resident.
__host__ __device__ constexpr int conv_b_stride(int cout) { return cout * KB * 2 < 1024 ? 1024 : cout * KB * 2; }

struct ConvArgs {
    CUtensorMap tin;               // [H Wp][Cin] bf16, box (32, 128)
    CUtensorMap twt;               // [9 Cout][Cin] bf16, box (32, Cout)
    const float* bias;             // [Cout]
    void* out;                     // [H Wp][Cout], bf16 or f32
    const __nv_bfloat16* mask;     // [H Wp][Cout] or NULL: zero the outputs where mask <= 0
    int out_f32, relu;
    int H, W, Wp, NP, Cin, Cout;
    uint32_t idesc;
    unsigned* err;
};

__global__ void __launch_bounds__(CONV_THREADS, 1) conv3x3_tc_kernel(const __grid_constant__ ConvArgs a) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sA = smem;
    uint8_t* sB = smem + CONV_STAGES * A_TILE_BYTES;
    const int b_stride = conv_b_stride(a.Cout);   // bytes of a stage's weight tile
    uint64_t* full = reinterpret_cast<uint64_t*>(sB + CONV_STAGES * b_stride);
    uint64_t* empty = full + CONV_STAGES;
    uint64_t* done = empty + CONV_STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
    __shared__ int s_fail;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int p0 = blockIdx.x * TILE_PIX;
    const int cblocks = a.Cin / KB, nkb = 9 * cblocks;
    const uint32_t tcols = a.Cout < 32 ? 32u : (uint32_t)a.Cout;
    const uint32_t b_bytes = (uint32_t)a.Cout * KB * 2;

    if (threadIdx.x == 0) {
        s_fail = 0;
        for (int i = 0; i < CONV_STAGES; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        mbar_init(done, 1);
        fence_mbar_init();
    }
    if (warp == 1) tmem_alloc(tmem_slot, tcols);
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {   // ---- TMA producer ----
            for (int kb = 0; kb < nkb; ++kb) {
                const int st = kb % CONV_STAGES, round = kb / CONV_STAGES;
                if (round > 0 && !mbar_wait(&empty[st], (round - 1) & 1)) {
                    s_fail = 1;
                    break;
                }
                const int tap = kb / cblocks, cb = kb - tap * cblocks;
                const int off = (tap / 3 - 1) * a.Wp + (tap % 3 - 1);
                mbar_expect_tx(&full[st], A_TILE_BYTES + b_bytes);
                tma_load_2d(sA + st * A_TILE_BYTES, &a.tin, &full[st], cb * KB, p0 + off);
                tma_load_2d(sB + st * b_stride, &a.twt, &full[st], cb * KB, tap * a.Cout);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {   // ---- MMA issuer ----
            for (int kb = 0; kb < nkb; ++kb) {
                const int st = kb % CONV_STAGES, round = kb / CONV_STAGES;
                if (!mbar_wait(&full[st], round & 1)) {
                    s_fail = 1;
                    break;
                }
                fence_after();
                const uint32_t a_base = smem_u32(sA + st * A_TILE_BYTES);
                const uint32_t b_base = smem_u32(sB + st * b_stride);
#pragma unroll
                for (int kk = 0; kk < KB / 16; ++kk)
                    umma_bf16(tmem, umma_desc_sw64(a_base + kk * 32), umma_desc_sw64(b_base + kk * 32), a.idesc,
                              (kb | kk) ? 1u : 0u);
                umma_commit(&empty[st]);   // frees the stage once these MMAs have read it
            }
            umma_commit(done);
        }
    } else {   // ---- epilogue: warps 2..5 read TMEM lanes 32 (warp % 4) .. +31 ----
        const int quarter = warp & 3;
        const int p = p0 + quarter * 32 + lane;
        const bool ok = mbar_wait(done, 0);
        if (!ok) s_fail = 1;
        fence_after();
        if (ok) {
            const int x = p % a.Wp;
            const bool live = p < a.NP, pad = x >= a.W;
            const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
            for (int c0 = 0; c0 < a.Cout; c0 += 16) {
                uint32_t r[16];
                tmem_ld16(tmem + lane_base + c0, r);
                tmem_wait_ld();
                float v[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    float t = __uint_as_float(r[j]) + __ldg(a.bias + c0 + j);
                    if (a.relu) t = fmaxf(t, 0.0f);
                    v[j] = pad ? 0.0f : t;
                }
                if (!live) continue;
                if (a.mask) {   // adjoint of a ReLU: the gradient passes where the activation is positive
                    const uint4* mp = reinterpret_cast<const uint4*>(a.mask + (size_t)p * a.Cout + c0);
                    const uint4 mw[2] = {__ldg(mp), __ldg(mp + 1)};
                    const __nv_bfloat16* mb = reinterpret_cast<const __nv_bfloat16*>(mw);
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (!(__bfloat162float(mb[j]) > 0.0f)) v[j] = 0.0f;
                }
                if (a.out_f32) {
                    float4* o = reinterpret_cast<float4*>(static_cast<float*>(a.out) + (size_t)p * a.Cout + c0);
#pragma unroll
                    for (int j = 0; j < 4; ++j) o[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                } else {
                    uint4 w[2];
                    uint32_t* wp = reinterpret_cast<uint32_t*>(w);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
                        wp[j] = *reinterpret_cast<uint32_t*>(&h);
                    }
                    uint4* o = reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(a.out) + (size_t)p * a.Cout + c0);
                    o[0] = w[0];
                    o[1] = w[1];
                }
            }
        }
    }
    fence_before();
    __syncthreads();
    if (s_fail && threadIdx.x == 0) atomicOr(a.err, 1u);
    if (warp == 1) {
        fence_after();
        tmem_dealloc(tmem, tcols);
    }
}

constexpr size_t conv_smem_bytes(int cout = 128) {
    return 1024 + CONV_STAGES * (A_TILE_BYTES + conv_b_stride(cout)) + (2 * CONV_STAGES + 1) * 8 + 16;
}

// ---------------------------------------------------------------------------
// Weight gradient on the tensor cores: for one tap,
//     dW[tap][co][ci] = sum_p g[p][co] x[p + off(tap)][ci]
// is a GEMM D = A B^T over K = pixels with A[co][p] = g[p][co] and
// B[ci][p] = x[p + off][ci]. Both operands arrive from the NHWC arrays as
// TMA boxes of 32 channels x 64 pixels (64-byte rows of channels, 64-byte
// swizzle): channel-contiguous, i.e. MN-major, so the instruction descriptor
// sets both major bits and the shared-memory descriptors use the canonical
// MN-major 64-byte-swizzle layout ((4, m), (8, k)) : ((1, LBO), (4, SBO)) in
// 16-byte units: a 32-channel group is one 64-byte row of a box, the next
// group (the next box) LBO = 4 KiB further, 8-pixel row groups SBO = 512 bytes
// apart. M = 128 output channels, N = Cin.
// A CTA sums one chunk of pixels for one tap in TMEM (f32) and adds its
// partial to dW with float32 atomics. (The bias gradient comes with g: the
// gradient kernels below.) Pixels past the level and shifted rows outside it are zero
// fill; the pad column of g is zero.
// ---------------------------------------------------------------------------
constexpr int WG_PIX = 64;                                  // pixels per stage
constexpr int WG_ALIGN = 32;                                // chunks are multiples of this
constexpr int WG_BOX = 32 * WG_PIX * 2;                     // one 32-channel x 64-pixel box: 4 KiB
constexpr int WG_A_BYTES = 4 * WG_BOX;                      // 128 channels of g
constexpr int WG_B_MAX = 4 * WG_BOX;                        // up to 128 channels of x
constexpr int WG_STAGES = 4;

struct WgradArgs {
    CUtensorMap tg;                // g: [NP][CGp] bf16, box (32 channels, 64 pixels)
    CUtensorMap tx;                // x: [NP][Cin] bf16, box (32, 64)
    float* dw;                     // [9][Cout][Cin] float32, accumulated into
    int Cout, CGp, Cin, Wp, NP;    // CGp: channels of g, Cout or the 32 it is padded to
    int chunk;                     // pixels per CTA (a multiple of WG_ALIGN)
    uint32_t idesc;
    long long wait_limit;
    unsigned* err;
};

// MN-major shared-memory descriptor, 64-byte swizzle (version 1, sm_100).
__device__ __forceinline__ uint64_t umma_desc_mn_sw64(uint32_t saddr, uint32_t lbo_bytes) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3fff);
    d |= (uint64_t)((lbo_bytes >> 4) & 0x3fff) << 16;   // next 32-channel group
    d |= (uint64_t)(512 >> 4) << 32;                     // next 8-pixel row group
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;
    return d;
}

__host__ __device__ constexpr uint32_t idesc_bf16_mn(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((uint32_t)(N >> 3) << 17) |
           ((uint32_t)(M >> 4) << 24);
}

__global__ void __launch_bounds__(CONV_THREADS, 1) conv_wgrad_tc_kernel(const __grid_constant__ WgradArgs a) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sA = smem;
    uint8_t* sB = smem + WG_STAGES * WG_A_BYTES;
    uint64_t* full = reinterpret_cast<uint64_t*>(sB + WG_STAGES * WG_B_MAX);
    uint64_t* empty = full + WG_STAGES;
    uint64_t* done = empty + WG_STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
    __shared__ int s_fail;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tap = blockIdx.y, off = (tap / 3 - 1) * a.Wp + (tap % 3 - 1);
    const int pa = blockIdx.x * a.chunk;
    const int pixels = min(a.NP, pa + a.chunk) - pa, nkb = (pixels + WG_PIX - 1) / WG_PIX;
    const int nbx = a.Cin / 32;                              // boxes of x per stage
    const uint32_t tcols = (uint32_t)a.Cin;                  // 32, 64 or 128 columns
    const uint32_t bytes = (uint32_t)(a.CGp / 32 + nbx) * WG_BOX;

    if (threadIdx.x == 0) {
        s_fail = 0;
        for (int i = 0; i < WG_STAGES; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        mbar_init(done, 1);
        fence_mbar_init();
    }
    if (warp == 1) tmem_alloc(tmem_slot, tcols);
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {   // ---- TMA producer ----
            for (int kb = 0; kb < nkb; ++kb) {
                const int st = kb % WG_STAGES, round = kb / WG_STAGES;
                if (round > 0 && !mbar_wait(&empty[st], (round - 1) & 1, a.wait_limit)) {
                    s_fail = 1;
                    break;
                }
                const int p = pa + kb * WG_PIX;
                mbar_expect_tx(&full[st], bytes);
                for (int c = 0; c < a.CGp / 32; ++c)   // channels 32c .. 32c + 31 of g
                    tma_load_2d(sA + st * WG_A_BYTES + c * WG_BOX, &a.tg, &full[st], 32 * c, p);
                for (int c = 0; c < nbx; ++c)
                    tma_load_2d(sB + st * WG_B_MAX + c * WG_BOX, &a.tx, &full[st], 32 * c, p + off);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {   // ---- MMA issuer ----
            for (int kb = 0; kb < nkb; ++kb) {
                const int st = kb % WG_STAGES, round = kb / WG_STAGES;
                if (!mbar_wait(&full[st], round & 1, a.wait_limit)) {
                    s_fail = 1;
                    break;
                }
                fence_after();
                const uint32_t a_base = smem_u32(sA + st * WG_A_BYTES);
                const uint32_t b_base = smem_u32(sB + st * WG_B_MAX);
                // 16 pixels (two 8-row groups) per MMA, up to the chunk's end
                const int nkk = min(WG_PIX, (pixels - kb * WG_PIX + 15) / 16 * 16) / 16;
                for (int kk = 0; kk < nkk; ++kk)
                    umma_bf16(tmem, umma_desc_mn_sw64(a_base + kk * 1024, WG_BOX),
                              umma_desc_mn_sw64(b_base + kk * 1024, WG_BOX), a.idesc, (kb | kk) ? 1u : 0u);
                umma_commit(&empty[st]);
            }
            umma_commit(done);
        }
    } else {   // ---- epilogue: warps 2..5 read TMEM lanes 32 (warp % 4) .. +31 (output channel) ----
        const int quarter = warp & 3;
        const int co = quarter * 32 + lane;
        const bool ok = nkb > 0 && mbar_wait(done, 0, a.wait_limit);
        if (nkb > 0 && !ok) s_fail = 1;
        fence_after();
        if (ok) {
            const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
            for (int c0 = 0; c0 < a.Cin; c0 += 16) {
                uint32_t r[16];
                tmem_ld16(tmem + lane_base + c0, r);
                tmem_wait_ld();
                if (co < a.Cout) {
                    float* d = a.dw + ((size_t)tap * a.Cout + co) * a.Cin + c0;
#pragma unroll
                    for (int j = 0; j < 16; ++j) atomicAdd(d + j, __uint_as_float(r[j]));
                }
            }
        }
    }
    fence_before();
    __syncthreads();
    if (s_fail && threadIdx.x == 0) atomicOr(a.err, 1u);
    if (warp == 1) {
        fence_after();
        tmem_dealloc(tmem, tcols);
    }
}

constexpr size_t wgrad_smem_bytes() {
    return 1024 + WG_STAGES * (WG_A_BYTES + WG_B_MAX) + (2 * WG_STAGES + 1) * 8 + 16;
}

// ---------------------------------------------------------------------------
// Element-wise kernels
// ---------------------------------------------------------------------------
struct Level {
    int H, W, Wp, NP;
};

__device__ __forceinline__ uint32_t pack_bf2(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}

__device__ __forceinline__ void unpack_bf8(uint4 u, float (&v)[8]) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 f = __bfloat1622float2(h[j]);
        v[2 * j] = f.x;
        v[2 * j + 1] = f.y;
    }
}

__device__ __forceinline__ uint4 pack_bf8(const float (&v)[8]) {
    return make_uint4(pack_bf2(v[0], v[1]), pack_bf2(v[2], v[3]), pack_bf2(v[4], v[5]), pack_bf2(v[6], v[7]));
}

struct PackArgs {
    const double* f1[9];           // ro, jx, jy, jz, Ex, Ey, Bx, By, Bz at t-1
    const double* f2[9];           // the same at t-2
    const double* scale;           // [23] device: input channel scales, then output scales
    double* partial;               // [STAT_BLOCKS][18] sums of squares
    double mult[23];               // multipliers of the scales
    __nv_bfloat16* x0;             // [NP][32]
    Level L;
};

// Per-sample channel statistics: partial sums of f1_c^2 and (f1_c - f2_c)^2
// per block, then one block adds them in a fixed order (deterministic) and
// sets scale_c = mult_c rms_c (1 where rms_c = 0). The output scale, shared
// by the 5 predicted fields, is the root mean square of the step
// differences of Ex, Ey, Bx, By, Bz (times the field's multiplier): the
// first-pass correction is of the order of one step's change.
constexpr int STAT_BLOCKS = 296;

__global__ void __launch_bounds__(256) stats_kernel(const __grid_constant__ PackArgs a) {
    double s[18];
#pragma unroll
    for (int c = 0; c < 18; ++c) s[c] = 0.0;
    const int n = a.L.H * a.L.W;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
#pragma unroll
        for (int c = 0; c < 9; ++c) {
            const double u1 = __ldg(a.f1[c] + i), d = u1 - __ldg(a.f2[c] + i);
            s[c] += u1 * u1;
            s[9 + c] += d * d;
        }
    __shared__ double ws[8][18];
#pragma unroll
    for (int c = 0; c < 18; ++c) {
        double v = s[c];
#pragma unroll
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5][c] = v;
    }
    __syncthreads();
    if (threadIdx.x < 18) {
        double v = 0.0;
        for (int w = 0; w < 8; ++w) v += ws[w][threadIdx.x];
        a.partial[blockIdx.x * 18 + threadIdx.x] = v;
    }
}

__global__ void scale_final_kernel(const __grid_constant__ PackArgs a) {
    const int c = threadIdx.x;
    double* scale = const_cast<double*>(a.scale);
    __shared__ double rms[18];
    if (c < 18) {
        double v = 0.0;
        for (int b = 0; b < STAT_BLOCKS; ++b) v += a.partial[b * 18 + c];
        rms[c] = sqrt(v / ((double)a.L.H * a.L.W));
        scale[c] = rms[c] > 0 ? a.mult[c] * rms[c] : 1.0;
    }
    __syncthreads();
    if (c < 5) {
        // differences of Ex, Ey, Bx, By, Bz: channels 13..17
        double m2 = 0.0;
        for (int f = 13; f < 18; ++f) m2 += rms[f] * rms[f];
        const double o = sqrt(m2 / 5.0);
        scale[18 + c] = o > 0 ? a.mult[18 + c] * o : 1.0;
    }
}

// x0[p] = (f1 / s_c, (f1 - f2) / d_c, log10(s_c) / 4, 0 ...), zero in the
// pad column: 9 fields, 9 differences, 9 constant channels that carry the
// absolute field levels the per-sample normalisation removes.
__global__ void pack_kernel(const __grid_constant__ PackArgs a) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.L.NP) return;
    const int y = p / a.L.Wp, x = p - y * a.L.Wp;
    float v[32];
#pragma unroll
    for (int c = 0; c < 32; ++c) v[c] = 0.0f;
    if (x < a.L.W) {
        const size_t i = (size_t)y * a.L.W + x;
#pragma unroll
        for (int c = 0; c < 9; ++c) {
            const double u1 = __ldg(a.f1[c] + i), u2 = __ldg(a.f2[c] + i);
            v[c] = (float)(u1 * (1.0 / a.scale[c]));
            v[9 + c] = (float)((u1 - u2) * (1.0 / a.scale[9 + c]));
            v[18 + c] = (float)(log10(a.scale[c]) * 0.25);
        }
    }
    uint4* o = reinterpret_cast<uint4*>(a.x0 + (size_t)p * 32);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        float w[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) w[j] = v[8 * q + j];
        o[q] = pack_bf8(w);
    }
}

// 2 x 2 average pooling (ceil mode: border cells average their valid
// children). One thread per (output pixel, 8 channels).
__global__ void pool_kernel(const __nv_bfloat16* __restrict__ in, Level li, __nv_bfloat16* __restrict__ out, Level lo,
                            int C) {
    const int groups = C / 8;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)lo.NP * groups) return;
    const int p = (int)(t / groups), g = (int)(t - (long long)p * groups);
    const int Y = p / lo.Wp, X = p - Y * lo.Wp;
    float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (X < lo.W) {
        int cnt = 0;
        for (int dy = 0; dy < 2; ++dy)
            for (int dx = 0; dx < 2; ++dx) {
                const int y = 2 * Y + dy, x = 2 * X + dx;
                if (y >= li.H || x >= li.W) continue;
                float v[8];
                unpack_bf8(*reinterpret_cast<const uint4*>(in + ((size_t)y * li.Wp + x) * C + 8 * g), v);
#pragma unroll
                for (int j = 0; j < 8; ++j) s[j] += v[j];
                ++cnt;
            }
        const float r = 1.0f / (float)cnt;
#pragma unroll
        for (int j = 0; j < 8; ++j) s[j] *= r;
    }
    *reinterpret_cast<uint4*>(out + (size_t)p * C + 8 * g) = pack_bf8(s);
}

// d = relu(up(u) + e): u at the coarse level, e and d at the fine level.
__global__ void upadd_relu_kernel(const __nv_bfloat16* __restrict__ u, Level lc, const __nv_bfloat16* __restrict__ e,
                                  __nv_bfloat16* __restrict__ d, Level lf, int C) {
    const int groups = C / 8;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)lf.NP * groups) return;
    const int p = (int)(t / groups), g = (int)(t - (long long)p * groups);
    const int y = p / lf.Wp, x = p - y * lf.Wp;
    float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (x < lf.W) {
        float a[8], b[8];
        unpack_bf8(*reinterpret_cast<const uint4*>(u + ((size_t)(y >> 1) * lc.Wp + (x >> 1)) * C + 8 * g), a);
        unpack_bf8(*reinterpret_cast<const uint4*>(e + (size_t)p * C + 8 * g), b);
#pragma unroll
        for (int j = 0; j < 8; ++j) s[j] = fmaxf(a[j] + b[j], 0.0f);
    }
    *reinterpret_cast<uint4*>(d + (size_t)p * C + 8 * g) = pack_bf8(s);
}

// Fields Ex, Ey, Ez, Bx, By, Bz; the network's 5 outputs are Ex, Ey, Bx,
// By, Bz (field indices net_field(k)); Ez is extrapolated linearly.
__device__ __host__ constexpr int net_field(int k) { return k < 2 ? k : k + 1; }

struct OutArgs {
    const double* f1[6];           // Ex, Ey, Ez, Bx, By, Bz at t-1
    const double* f2[6];           // ... at t-2
    const double* first[6];        // target: first-pass fields at t (training; Ez unused)
    double* pred[6];               // prediction at t (inference)
    const double* scale;           // [23] device scales; the output scales at 18..
    const float* y;                // [NP][16]
    float* target;                 // [NP][16]
    Level L;
};

// pred = 2 f1 - f2 + scale * y (Ez: 2 f1 - f2)
__global__ void unpack_kernel(const __grid_constant__ OutArgs a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.L.H * a.L.W) return;
    const int yy = i / a.L.W, x = i - yy * a.L.W;
    const float* yp = a.y + ((size_t)yy * a.L.Wp + x) * 16;
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const int f = net_field(k);
        a.pred[f][i] = 2.0 * __ldg(a.f1[f] + i) - __ldg(a.f2[f] + i) + a.scale[18 + k] * (double)yp[k];
    }
    a.pred[2][i] = 2.0 * __ldg(a.f1[2] + i) - __ldg(a.f2[2] + i);
}

// target = (first - (2 f1 - f2)) / scale, zero elsewhere
__global__ void target_kernel(const __grid_constant__ OutArgs a) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.L.NP) return;
    const int yy = p / a.L.Wp, x = p - yy * a.L.Wp;
    float v[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) v[c] = 0.0f;
    if (x < a.L.W) {
        const size_t i = (size_t)yy * a.L.W + x;
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            const int f = net_field(k);
            v[k] = (float)((__ldg(a.first[f] + i) - (2.0 * __ldg(a.f1[f] + i) - __ldg(a.f2[f] + i))) / a.scale[18 + k]);
        }
    }
    float4* o = reinterpret_cast<float4*>(a.target + (size_t)p * 16);
#pragma unroll
    for (int q = 0; q < 4; ++q) o[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
}

// ---------------------------------------------------------------------------
// Backward data pass on the tensor cores. dL/dx of a 3x3 convolution is the
// 3x3 convolution of the output gradient g with the flipped, transposed
// weights, W'[tap][ci][co] = W[8 - tap][co][ci] (tap 8 - t is the opposite
// shift of tap t), so conv3x3_tc_kernel computes it: g is rounded to bf16
// (its channels padded with zeros to a multiple of 32, zero in the pad
// column), the accumulation is f32 in TMEM, and the epilogue applies the
// ReLU adjoint of the layer's input.
// ---------------------------------------------------------------------------

// wt[tap][ci][co] = w[8 - tap][co][ci] (co < CG), 0 for CG <= co < CGp.
__global__ void flip_weights_kernel(const __nv_bfloat16* __restrict__ w, int CG, int CIN, int CGp,
                                    __nv_bfloat16* __restrict__ wt) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 9 * CIN * CGp) return;
    const int tap = t / (CIN * CGp), rem = t - tap * CIN * CGp, ci = rem / CGp, co = rem - ci * CGp;
    wt[t] = co < CG ? w[((size_t)(8 - tap) * CG + co) * CIN + ci] : __float2bfloat16_rn(0.0f);
}

// ---------------------------------------------------------------------------
// Training kernels: loss, pooling / upsampling / ReLU adjoints with the bias
// gradients, Adam
// ---------------------------------------------------------------------------

// The kernels that produce a layer's output gradient write it in bf16, the
// operand of both tensor-core passes (0 in the pad column and past CG
// channels), and add its sums over the pixels to the bias gradient db on the
// way: a thread has 8 channels of every few hundredth pixel, a CTA adds its
// sums by float32 atomics. (A separate bias kernel, 128 CTAs walking the
// float32 gradient pixel by pixel, took 970 of the 2200 us of a training
// sample at 641^2, a separate conversion 160.)
constexpr int GRAD_THREADS = 256;

// s[8] of every thread, thread t holding channel group t % G, summed over the
// CTA into db[0 .. 8 G). G = 4, 8 or 16.
__device__ __forceinline__ void add_bias_sums(float (&s)[8], int G, float* db) {
    __shared__ float ws[GRAD_THREADS / 32][128];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 16; o >= G; o >>= 1)
#pragma unroll
        for (int j = 0; j < 8; ++j) s[j] += __shfl_xor_sync(0xffffffffu, s[j], o);
    if (lane < G)
#pragma unroll
        for (int j = 0; j < 8; ++j) ws[warp][lane * 8 + j] = s[j];
    __syncthreads();
    if ((int)threadIdx.x < 8 * G) {
        float v = 0.0f;
#pragma unroll
        for (int w = 0; w < GRAD_THREADS / 32; ++w) v += ws[w][threadIdx.x];
        atomicAdd(db + threadIdx.x, v);
    }
}

__device__ __forceinline__ void load8(const float* p, float (&v)[8]) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

// Mean squared error over the 5 used channels of the H x W pixels and its
// gradient: g[p][0 .. 32) = dL/dy, a thread per pixel.
__global__ void __launch_bounds__(GRAD_THREADS) loss_kernel(const float* __restrict__ y, const float* __restrict__ t,
                                                            __nv_bfloat16* __restrict__ g, Level L, float* loss,
                                                            float* __restrict__ db) {
    const float inv = 1.0f / (5.0f * (float)L.H * (float)L.W);
    float sq = 0.0f, s[5] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    for (int p = blockIdx.x * GRAD_THREADS + threadIdx.x; p < L.NP; p += gridDim.x * GRAD_THREADS) {
        float v[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        if (p % L.Wp < L.W) {
            float a[8], b[8];
            load8(y + (size_t)p * 16, a);
            load8(t + (size_t)p * 16, b);
#pragma unroll
            for (int c = 0; c < 5; ++c) {
                const float d = a[c] - b[c];
                sq += d * d;
                v[c] = 2.0f * d * inv;
                s[c] += v[c];
            }
        }
        uint4* o = reinterpret_cast<uint4*>(g + (size_t)p * 32);
        const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
        o[0] = pack_bf8(v);
        o[1] = zero;
        o[2] = zero;
        o[3] = zero;
    }
    __shared__ float ws[GRAD_THREADS / 32][6];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        sq += __shfl_xor_sync(0xffffffffu, sq, o);
#pragma unroll
        for (int c = 0; c < 5; ++c) s[c] += __shfl_xor_sync(0xffffffffu, s[c], o);
    }
    if (lane == 0) {
#pragma unroll
        for (int c = 0; c < 5; ++c) ws[warp][c] = s[c];
        ws[warp][5] = sq;
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        float v = 0.0f;
#pragma unroll
        for (int w = 0; w < GRAD_THREADS / 32; ++w) v += ws[w][threadIdx.x];
        if (threadIdx.x < 5) atomicAdd(db + threadIdx.x, v);
        else atomicAdd(loss, v * inv);
    }
}

// out = bf16(g), C channels.
__global__ void __launch_bounds__(GRAD_THREADS) grad_bf16_kernel(const float* __restrict__ g, __nv_bfloat16* __restrict__ out,
                                                                 Level L, int C, float* __restrict__ db) {
    const int G = C / 8, c = threadIdx.x % G * 8, per = GRAD_THREADS / G;
    float s[8] = {};
    for (int p = blockIdx.x * per + threadIdx.x / G; p < L.NP; p += gridDim.x * per) {
        float v[8] = {};
        if (p % L.Wp < L.W) {
            load8(g + (size_t)p * C + c, v);
#pragma unroll
            for (int j = 0; j < 8; ++j) s[j] += v[j];
        }
        *reinterpret_cast<uint4*>(out + (size_t)p * C + c) = pack_bf8(v);
    }
    add_bias_sums(s, G, db);
}

// out[Y][X][c] = sum of g_d over the valid fine children (adjoint of the
// nearest-neighbour upsampling).
__global__ void __launch_bounds__(GRAD_THREADS) downsum_kernel(const float* __restrict__ gd, Level lf,
                                                               __nv_bfloat16* __restrict__ out, Level lc, int C,
                                                               float* __restrict__ db) {
    const int G = C / 8, c = threadIdx.x % G * 8, per = GRAD_THREADS / G;
    float s[8] = {};
    for (int p = blockIdx.x * per + threadIdx.x / G; p < lc.NP; p += gridDim.x * per) {
        const int Y = p / lc.Wp, X = p - Y * lc.Wp;
        float v[8] = {};
        if (X < lc.W) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int y = 2 * Y + k / 2, x = 2 * X + k % 2;
                if (y < lf.H && x < lf.W) {
                    float w[8];
                    load8(gd + ((size_t)y * lf.Wp + x) * C + c, w);
#pragma unroll
                    for (int j = 0; j < 8; ++j) v[j] += w[j];
                }
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) s[j] += v[j];
        }
        *reinterpret_cast<uint4*>(out + (size_t)p * C + c) = pack_bf8(v);
    }
    add_bias_sums(s, G, db);
}

// out = (g_e + g_p[parent] / children(parent)) * (e > 0) (adjoint of the
// average pooling, plus the skip gradient in g_e, through the ReLU).
__global__ void __launch_bounds__(GRAD_THREADS) pool_bwd_mask_kernel(const float* __restrict__ ge,
                                                                     const __nv_bfloat16* __restrict__ e, Level lf,
                                                                     const float* __restrict__ gp, Level lc, int C,
                                                                     __nv_bfloat16* __restrict__ out,
                                                                     float* __restrict__ db) {
    const int G = C / 8, c = threadIdx.x % G * 8, per = GRAD_THREADS / G;
    float s[8] = {};
    for (int p = blockIdx.x * per + threadIdx.x / G; p < lf.NP; p += gridDim.x * per) {
        const int y = p / lf.Wp, x = p - y * lf.Wp;
        float v[8] = {};
        if (x < lf.W) {
            const int Y = y >> 1, X = x >> 1;
            const int cnt = (min(2 * Y + 2, lf.H) - 2 * Y) * (min(2 * X + 2, lf.W) - 2 * X);
            float w[8], act[8];
            load8(ge + (size_t)p * C + c, v);
            load8(gp + ((size_t)Y * lc.Wp + X) * C + c, w);
            unpack_bf8(__ldg(reinterpret_cast<const uint4*>(e + (size_t)p * C + c)), act);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                v[j] = act[j] > 0.0f ? v[j] + w[j] / (float)cnt : 0.0f;
                s[j] += v[j];
            }
        }
        *reinterpret_cast<uint4*>(out + (size_t)p * C + c) = pack_bf8(v);
    }
    add_bias_sums(s, G, db);
}

// Adam on the float32 master parameters; refreshes the bf16 copy.
__global__ void adam_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, __nv_bfloat16* __restrict__ pb, long long n, float lr, float b1,
                            float b2, float eps, float c1, float c2) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    p[i] = pi;
    pb[i] = __float2bfloat16_rn(pi);
}

__global__ void to_bf16_kernel(const float* __restrict__ p, __nv_bfloat16* __restrict__ pb, long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) pb[i] = __float2bfloat16_rn(p[i]);
}

}  // namespace

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
namespace {

struct LayerDef {
    int cin, cout, level, relu, out_f32;
};
// conv1 .. conv6 (see the network at the top of this file)
constexpr LayerDef LAYERS[NLAYERS] = {{32, 32, 0, 1, 0},  {32, 64, 1, 1, 0},  {64, 128, 2, 1, 0},
                                      {128, 64, 2, 0, 0}, {64, 32, 1, 0, 0},  {32, 16, 0, 0, 1}};

long long layer_wsize(int l) { return 9LL * LAYERS[l].cout * LAYERS[l].cin; }

long long param_offsets(long long* w_off, long long* b_off) {
    long long o = 0;
    for (int l = 0; l < NLAYERS; ++l) {
        if (w_off) w_off[l] = o;
        o += layer_wsize(l);
        if (b_off) b_off[l] = o;
        o += LAYERS[l].cout;
    }
    return o;
}

int make_map_2d(CUtensorMap* m, const void* base, long long rows, int cols, int box_rows) {
    auto enc = tc_get_encode();
    if (!enc) return LC3D_ERR_CUDA;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
    cuuint32_t box[2] = {(cuuint32_t)KB, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? LC3D_OK : LC3D_ERR_CUDA;
}

unsigned blocks_for(long long n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

struct lc3d_predictor {
    int device = 0, N = 0;
    Level lv[3];
    long long np = 0, w_off[NLAYERS], b_off[NLAYERS];
    float *params = nullptr, *grad = nullptr, *adam_m = nullptr, *adam_v = nullptr;
    __nv_bfloat16* wbf = nullptr;
    int adam_t = 0;
    // activations (bf16 NHWC) and the float32 output / target
    __nv_bfloat16 *x0 = nullptr, *e1 = nullptr, *p1 = nullptr, *e2 = nullptr, *p2 = nullptr, *e3 = nullptr,
                  *u3 = nullptr, *d2 = nullptr, *u2 = nullptr, *d1 = nullptr;
    float *y = nullptr, *target = nullptr;
    // gradients (float32 NHWC)
    float *g_d1 = nullptr, *g_d2 = nullptr, *g_e3 = nullptr, *g_p2 = nullptr, *g_p1 = nullptr;
    // tensor-core backward passes: the bf16 output gradients of two layers,
    // the flipped transposed bf16 weights of every layer, zeros for the bias, and the convolution arguments of each layer's pass
    __nv_bfloat16* g_bf[2] = {nullptr, nullptr};   // layer l uses g_bf[l & 1]
    __nv_bfloat16* wt = nullptr;
    long long wt_off[NLAYERS];
    float* zero_bias = nullptr;
    ConvArgs bconv[NLAYERS];
    WgradArgs wg[NLAYERS];         // tensor-core weight gradient of each layer
    dim3 wg_grid[NLAYERS];
    cudaStream_t wg_stream = nullptr;              // the weight-gradient passes' stream
    cudaEvent_t ev_grad[NLAYERS] = {}, ev_wg[NLAYERS] = {};   // layer l's g_bf written; read by its weight pass
    unsigned* err = nullptr;       // device word: a wait ran out (this object's own, not a context's flag words)
    double* scale = nullptr;       // [23] per-sample channel scales (device)
    double* partial = nullptr;     // [STAT_BLOCKS][18]
    double mult[23];               // scale multipliers (host-set)
    ConvArgs conv[NLAYERS];
    std::vector<void*> allocs;
};

namespace {

template <typename T>
int dalloc(lc3d_predictor* P, T** p, size_t count) {
    void* q = nullptr;
    LC3D_CUDA_TRY(cudaMalloc(&q, count * sizeof(T)));
    LC3D_CUDA_TRY(cudaMemset(q, 0, count * sizeof(T)));
    P->allocs.push_back(q);
    *p = static_cast<T*>(q);
    return LC3D_OK;
}

int setup_conv(lc3d_predictor* P, int l, const __nv_bfloat16* in, void* out) {
    const LayerDef& d = LAYERS[l];
    const Level& L = P->lv[d.level];
    ConvArgs& a = P->conv[l];
    memset(&a, 0, sizeof(a));
    LC3D_TRY(make_map_2d(&a.tin, in, L.NP, d.cin, TILE_PIX));
    LC3D_TRY(make_map_2d(&a.twt, P->wbf + P->w_off[l], 9LL * d.cout, d.cin, d.cout));
    a.bias = P->params + P->b_off[l];
    a.out = out;
    a.out_f32 = d.out_f32;
    a.relu = d.relu;
    a.H = L.H; a.W = L.W; a.Wp = L.Wp; a.NP = L.NP;
    a.Cin = d.cin; a.Cout = d.cout;
    a.idesc = idesc_bf16(TILE_PIX, d.cout);
    a.err = P->err;
    return LC3D_OK;
}

int run_conv(lc3d_predictor* P, int l, cudaStream_t s) {
    const ConvArgs& a = P->conv[l];
    conv3x3_tc_kernel<<<blocks_for(a.NP, TILE_PIX), CONV_THREADS, conv_smem_bytes(a.Cout), s>>>(a);
    LC3D_CUDA_TRY(cudaGetLastError());
    return LC3D_OK;
}

// Output-gradient channels of layer l as the tensor-core pass reads them.
int grad_channels(int l) { return LAYERS[l].cout < KB ? KB : LAYERS[l].cout; }

int setup_bconv(lc3d_predictor* P, int l) {
    const LayerDef& d = LAYERS[l];
    const Level& L = P->lv[d.level];
    const int CGp = grad_channels(l);
    ConvArgs& a = P->bconv[l];
    memset(&a, 0, sizeof(a));
    LC3D_TRY(make_map_2d(&a.tin, P->g_bf[l & 1], L.NP, CGp, TILE_PIX));
    LC3D_TRY(make_map_2d(&a.twt, P->wt + P->wt_off[l], 9LL * d.cin, CGp, d.cin));
    a.bias = P->zero_bias;
    a.out_f32 = 1;
    a.relu = 0;
    a.H = L.H; a.W = L.W; a.Wp = L.Wp; a.NP = L.NP;
    a.Cin = CGp; a.Cout = d.cin;
    a.idesc = idesc_bf16(TILE_PIX, d.cin);
    a.err = P->err;
    return LC3D_OK;
}

int setup_wgrad(lc3d_predictor* P, int l, const __nv_bfloat16* x) {
    const LayerDef& d = LAYERS[l];
    const Level& L = P->lv[d.level];
    WgradArgs& a = P->wg[l];
    memset(&a, 0, sizeof(a));
    LC3D_TRY(make_map_2d(&a.tg, P->g_bf[l & 1], L.NP, grad_channels(l), WG_PIX));
    LC3D_TRY(make_map_2d(&a.tx, x, L.NP, d.cin, WG_PIX));
    a.dw = P->grad + P->w_off[l];
    a.Cout = d.cout;
    a.CGp = grad_channels(l);
    a.Cin = d.cin;
    a.Wp = L.Wp;
    a.NP = L.NP;
    // 16 pixel chunks per tap: 9 x 16 CTAs
    const int chunks = (int)std::min<long long>(16, (L.NP + WG_ALIGN - 1) / WG_ALIGN);
    a.chunk = (int)(((L.NP + chunks - 1) / chunks + WG_ALIGN - 1) / WG_ALIGN * WG_ALIGN);
    P->wg_grid[l] = dim3((L.NP + a.chunk - 1) / a.chunk, 9);
    a.idesc = idesc_bf16_mn(128, d.cin);
    a.wait_limit = WAIT_LIMIT;
    a.err = P->err;
    return LC3D_OK;
}

// dW of layer l from its output gradient in g_bf.
int bwd_weights_tc(lc3d_predictor* P, int l, cudaStream_t s) {
    const WgradArgs& a = P->wg[l];
    conv_wgrad_tc_kernel<<<P->wg_grid[l], CONV_THREADS, wgrad_smem_bytes(), s>>>(a);
    LC3D_CUDA_TRY(cudaGetLastError());
    return LC3D_OK;
}

// dx = dL/d(input of layer l) from g_bf, zeroed where mask <= 0.
int bwd_data_tc(lc3d_predictor* P, int l, const __nv_bfloat16* mask, float* dx, cudaStream_t s) {
    ConvArgs a = P->bconv[l];
    a.out = dx;
    a.mask = mask;
    conv3x3_tc_kernel<<<blocks_for(a.NP, TILE_PIX), CONV_THREADS, conv_smem_bytes(a.Cout), s>>>(a);
    LC3D_CUDA_TRY(cudaGetLastError());
    return LC3D_OK;
}

int forward(lc3d_predictor* P, cudaStream_t s) {
    const Level *l0 = &P->lv[0], *l1 = &P->lv[1], *l2 = &P->lv[2];
    LC3D_TRY(run_conv(P, 0, s));
    pool_kernel<<<blocks_for((long long)l1->NP * 4, 256), 256, 0, s>>>(P->e1, *l0, P->p1, *l1, 32);
    LC3D_TRY(run_conv(P, 1, s));
    pool_kernel<<<blocks_for((long long)l2->NP * 8, 256), 256, 0, s>>>(P->e2, *l1, P->p2, *l2, 64);
    LC3D_TRY(run_conv(P, 2, s));
    LC3D_TRY(run_conv(P, 3, s));
    upadd_relu_kernel<<<blocks_for((long long)l1->NP * 8, 256), 256, 0, s>>>(P->u3, *l2, P->e2, P->d2, *l1, 64);
    LC3D_TRY(run_conv(P, 4, s));
    upadd_relu_kernel<<<blocks_for((long long)l0->NP * 4, 256), 256, 0, s>>>(P->u2, *l1, P->e1, P->d1, *l0, 32);
    LC3D_TRY(run_conv(P, 5, s));
    LC3D_CUDA_TRY(cudaGetLastError());
    return LC3D_OK;
}

int backward(lc3d_predictor* P, float* loss, cudaStream_t s) {
    const Level &l0 = P->lv[0], &l1 = P->lv[1], &l2 = P->lv[2];
    LC3D_CUDA_TRY(cudaMemsetAsync(P->grad, 0, (size_t)P->np * sizeof(float), s));
    // the flipped, transposed bf16 weights of the layers whose input gradient is needed
    for (int l = 1; l < NLAYERS; ++l) {
        const int n = 9 * LAYERS[l].cin * grad_channels(l);
        flip_weights_kernel<<<blocks_for(n, 256), 256, 0, s>>>(P->wbf + P->w_off[l], LAYERS[l].cout, LAYERS[l].cin,
                                                                grad_channels(l), P->wt + P->wt_off[l]);
    }
    LC3D_CUDA_TRY(cudaGetLastError());
    // Each layer: its output gradient in bf16 (g_bf[l & 1]) with the bias
    // gradient, then the data pass on this stream and the weight pass on a
    // second one: the weight pass waits on its MMAs with one CTA per SM, the
    // data pass on its loads with five (641^2: 866 -> 784 us a training
    // sample). A layer's gradient is written over the one of two layers before
    // once that layer's weight pass has read it.
    auto db = [&](int l) { return P->grad + P->b_off[l]; };
    auto grid = [&](const Level& L, int C) {   // CTAs of a gradient kernel: a few pixels per thread, six CTAs per SM at most
        return std::min(blocks_for((long long)L.NP * (C / 8), GRAD_THREADS * 4), 148u * 6);
    };
    auto before = [&](int l) -> int {   // g_bf[l & 1] is free
        if (l + 2 < NLAYERS) LC3D_CUDA_TRY(cudaStreamWaitEvent(s, P->ev_wg[l + 2], 0));
        return LC3D_OK;
    };
    auto weights = [&](int l) -> int {
        LC3D_CUDA_TRY(cudaEventRecord(P->ev_grad[l], s));
        LC3D_CUDA_TRY(cudaStreamWaitEvent(P->wg_stream, P->ev_grad[l], 0));
        LC3D_TRY(bwd_weights_tc(P, l, P->wg_stream));
        LC3D_CUDA_TRY(cudaEventRecord(P->ev_wg[l], P->wg_stream));
        return LC3D_OK;
    };
    // conv6: d1 -> y
    loss_kernel<<<grid(l0, 8), GRAD_THREADS, 0, s>>>(P->y, P->target, P->g_bf[1], l0, loss, db(5));
    LC3D_TRY(weights(5));
    LC3D_TRY(bwd_data_tc(P, 5, P->d1, P->g_d1, s));
    // conv5: d2 -> u2
    downsum_kernel<<<grid(l1, 32), GRAD_THREADS, 0, s>>>(P->g_d1, l0, P->g_bf[0], l1, 32, db(4));
    LC3D_TRY(weights(4));
    LC3D_TRY(bwd_data_tc(P, 4, P->d2, P->g_d2, s));
    // conv4: e3 -> u3
    LC3D_TRY(before(3));
    downsum_kernel<<<grid(l2, 64), GRAD_THREADS, 0, s>>>(P->g_d2, l1, P->g_bf[1], l2, 64, db(3));
    LC3D_TRY(weights(3));
    LC3D_TRY(bwd_data_tc(P, 3, P->e3, P->g_e3, s));
    // conv3: p2 -> e3
    LC3D_TRY(before(2));
    grad_bf16_kernel<<<grid(l2, 128), GRAD_THREADS, 0, s>>>(P->g_e3, P->g_bf[0], l2, 128, db(2));
    LC3D_TRY(weights(2));
    LC3D_TRY(bwd_data_tc(P, 2, nullptr, P->g_p2, s));
    // conv2: p1 -> e2
    LC3D_TRY(before(1));
    pool_bwd_mask_kernel<<<grid(l1, 64), GRAD_THREADS, 0, s>>>(P->g_d2, P->e2, l1, P->g_p2, l2, 64, P->g_bf[1], db(1));
    LC3D_TRY(weights(1));
    LC3D_TRY(bwd_data_tc(P, 1, nullptr, P->g_p1, s));
    // conv1: x0 -> e1
    LC3D_TRY(before(0));
    pool_bwd_mask_kernel<<<grid(l0, 32), GRAD_THREADS, 0, s>>>(P->g_d1, P->e1, l0, P->g_p1, l1, 32, P->g_bf[0], db(0));
    LC3D_TRY(weights(0));
    // the second stream is in order: its last pass ends the backward pass
    LC3D_CUDA_TRY(cudaStreamWaitEvent(s, P->ev_wg[0], 0));
    LC3D_CUDA_TRY(cudaGetLastError());
    return LC3D_OK;
}

struct PredDevice {
    int dev;
    explicit PredDevice(int d) {
        cudaGetDevice(&dev);
        cudaSetDevice(d);
    }
    ~PredDevice() { cudaSetDevice(dev); }
};

cudaStream_t St(void* s) { return static_cast<cudaStream_t>(s); }

}  // namespace

extern "C" {

long long lc3d_predictor_num_params(void) { return param_offsets(nullptr, nullptr); }

int lc3d_predictor_create(int grid_steps, int device, lc3d_predictor** out) {
    if (!out || grid_steps < 9 || grid_steps > 4097) return LC3D_ERR_PARAM;
    *out = nullptr;
    PredDevice g(device);
    lc3d_predictor* P = new lc3d_predictor();
    P->device = device;
    P->N = grid_steps;
    int H = grid_steps;
    for (int k = 0; k < 3; ++k) {
        P->lv[k] = Level{H, H, H + 1, H * (H + 1)};
        H = (H + 1) / 2;
    }
    P->np = param_offsets(P->w_off, P->b_off);
    for (int c = 0; c < 23; ++c) P->mult[c] = 1.0;
    const size_t n0 = P->lv[0].NP, n1 = P->lv[1].NP, n2 = P->lv[2].NP;
    int rc = LC3D_OK;
#define PA(ptr, cnt) \
    if (rc == LC3D_OK) rc = dalloc(P, &(ptr), (cnt))
    PA(P->params, P->np); PA(P->grad, P->np); PA(P->adam_m, P->np); PA(P->adam_v, P->np); PA(P->wbf, P->np);
    PA(P->x0, n0 * 32); PA(P->e1, n0 * 32); PA(P->p1, n1 * 32); PA(P->e2, n1 * 64); PA(P->p2, n2 * 64);
    PA(P->e3, n2 * 128); PA(P->u3, n2 * 64); PA(P->d2, n1 * 64); PA(P->u2, n1 * 32); PA(P->d1, n0 * 32);
    PA(P->y, n0 * 16); PA(P->target, n0 * 16);
    PA(P->g_d1, n0 * 32); PA(P->g_d2, n1 * 64); PA(P->g_e3, n2 * 128); PA(P->g_p2, n2 * 64); PA(P->g_p1, n1 * 32);
    PA(P->err, 1); PA(P->scale, 23); PA(P->partial, (size_t)STAT_BLOCKS * 18);
    {   // tensor-core backward data pass (layers 2..6; the input gradient of layer 1 is not needed)
        size_t gmax = 0;
        long long wtot = 0;
        for (int l = 0; l < NLAYERS; ++l) {
            P->wt_off[l] = wtot;
            gmax = std::max(gmax, (size_t)P->lv[LAYERS[l].level].NP * grad_channels(l));
            if (l == 0) continue;
            wtot += 9LL * LAYERS[l].cin * grad_channels(l);
        }
        PA(P->g_bf[0], gmax); PA(P->g_bf[1], gmax); PA(P->wt, (size_t)wtot); PA(P->zero_bias, 128);
    }
#undef PA
    if (rc == LC3D_OK) rc = setup_conv(P, 0, P->x0, P->e1);
    if (rc == LC3D_OK) rc = setup_conv(P, 1, P->p1, P->e2);
    if (rc == LC3D_OK) rc = setup_conv(P, 2, P->p2, P->e3);
    if (rc == LC3D_OK) rc = setup_conv(P, 3, P->e3, P->u3);
    if (rc == LC3D_OK) rc = setup_conv(P, 4, P->d2, P->u2);
    if (rc == LC3D_OK) rc = setup_conv(P, 5, P->d1, P->y);
    if (rc == LC3D_OK && cudaStreamCreateWithFlags(&P->wg_stream, cudaStreamNonBlocking) != cudaSuccess) rc = LC3D_ERR_CUDA;
    for (int l = 0; l < NLAYERS && rc == LC3D_OK; ++l)
        if (cudaEventCreateWithFlags(&P->ev_grad[l], cudaEventDisableTiming) != cudaSuccess ||
            cudaEventCreateWithFlags(&P->ev_wg[l], cudaEventDisableTiming) != cudaSuccess)
            rc = LC3D_ERR_CUDA;
    for (int l = 1; l < NLAYERS && rc == LC3D_OK; ++l) rc = setup_bconv(P, l);
    {   // the input activation of each layer, for its weight gradient
        const __nv_bfloat16* xin[NLAYERS] = {P->x0, P->p1, P->p2, P->e3, P->d2, P->d1};
        for (int l = 0; l < NLAYERS && rc == LC3D_OK; ++l) rc = setup_wgrad(P, l, xin[l]);
    }
    if (rc == LC3D_OK) {
        static bool attrs_set[64] = {};
        bool& attrs = attrs_set[device & 63];
        if (!attrs) {
            cudaFuncSetAttribute(conv3x3_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)conv_smem_bytes());
            cudaFuncSetAttribute(conv_wgrad_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)wgrad_smem_bytes());
            attrs = cudaGetLastError() == cudaSuccess;
            if (!attrs) rc = LC3D_ERR_CUDA;
        }
    }
    if (rc != LC3D_OK) {
        lc3d_predictor_destroy(P);
        return rc;
    }
    *out = P;
    return LC3D_OK;
}

int lc3d_predictor_destroy(lc3d_predictor* P) {
    if (!P) return LC3D_OK;
    PredDevice g(P->device);
    for (void* q : P->allocs) cudaFree(q);
    for (int l = 0; l < NLAYERS; ++l) {
        if (P->ev_grad[l]) cudaEventDestroy(P->ev_grad[l]);
        if (P->ev_wg[l]) cudaEventDestroy(P->ev_wg[l]);
    }
    if (P->wg_stream) cudaStreamDestroy(P->wg_stream);
    delete P;
    return LC3D_OK;
}

int lc3d_predictor_set_params(lc3d_predictor* P, const float* params, void* stream) {
    if (!P || !params) return LC3D_ERR_PARAM;
    PredDevice g(P->device);
    LC3D_CUDA_TRY(cudaMemcpyAsync(P->params, params, (size_t)P->np * sizeof(float), cudaMemcpyDeviceToDevice,
                                  St(stream)));
    to_bf16_kernel<<<blocks_for(P->np, 256), 256, 0, St(stream)>>>(P->params, P->wbf, P->np);
    LC3D_CUDA_TRY(cudaMemsetAsync(P->adam_m, 0, (size_t)P->np * sizeof(float), St(stream)));
    LC3D_CUDA_TRY(cudaMemsetAsync(P->adam_v, 0, (size_t)P->np * sizeof(float), St(stream)));
    P->adam_t = 0;
    LC3D_CUDA_TRY(cudaGetLastError());
    return LC3D_OK;
}

int lc3d_predictor_get_params(lc3d_predictor* P, float* params, void* stream) {
    if (!P || !params) return LC3D_ERR_PARAM;
    PredDevice g(P->device);
    LC3D_CUDA_TRY(cudaMemcpyAsync(params, P->params, (size_t)P->np * sizeof(float), cudaMemcpyDeviceToDevice,
                                  St(stream)));
    return LC3D_OK;
}

int lc3d_predictor_get_grad(lc3d_predictor* P, float* grad, void* stream) {
    if (!P || !grad) return LC3D_ERR_PARAM;
    PredDevice g(P->device);
    LC3D_CUDA_TRY(cudaMemcpyAsync(grad, P->grad, (size_t)P->np * sizeof(float), cudaMemcpyDeviceToDevice,
                                  St(stream)));
    return LC3D_OK;
}

int lc3d_predictor_set_scales(lc3d_predictor* P, const double* in_mult, const double* out_mult) {
    if (!P || !in_mult || !out_mult) return LC3D_ERR_PARAM;
    for (int c = 0; c < 18; ++c)
        if (!(in_mult[c] > 0) || !std::isfinite(in_mult[c])) return LC3D_ERR_PARAM;
    for (int c = 0; c < 5; ++c)
        if (!(out_mult[c] > 0) || !std::isfinite(out_mult[c])) return LC3D_ERR_PARAM;
    memcpy(P->mult, in_mult, 18 * sizeof(double));
    memcpy(P->mult + 18, out_mult, 5 * sizeof(double));
    return LC3D_OK;
}

int lc3d_predictor_pack(lc3d_predictor* P, const double* const* f1, const double* const* f2, void* stream) {
    if (!P || !f1 || !f2) return LC3D_ERR_PARAM;
    PackArgs a{};
    for (int c = 0; c < 9; ++c) {
        if (!f1[c] || !f2[c]) return LC3D_ERR_PARAM;
        a.f1[c] = f1[c];
        a.f2[c] = f2[c];
    }
    a.scale = P->scale;
    a.partial = P->partial;
    memcpy(a.mult, P->mult, sizeof(a.mult));
    a.x0 = P->x0;
    a.L = P->lv[0];
    PredDevice g(P->device);
    stats_kernel<<<STAT_BLOCKS, 256, 0, St(stream)>>>(a);
    scale_final_kernel<<<1, 32, 0, St(stream)>>>(a);
    pack_kernel<<<blocks_for(a.L.NP, 128), 128, 0, St(stream)>>>(a);
    LC3D_CUDA_TRY(cudaGetLastError());
    return LC3D_OK;
}

int lc3d_predictor_forward(lc3d_predictor* P, void* stream) {
    if (!P) return LC3D_ERR_PARAM;
    PredDevice g(P->device);
    return forward(P, St(stream));
}

static int out_args(lc3d_predictor* P, OutArgs* a, const double* const* f1, const double* const* f2, bool ez) {
    memset(a, 0, sizeof(*a));
    for (int f = 0; f < 6; ++f) {
        if ((f != 2 || ez) && (!f1[f] || !f2[f])) return LC3D_ERR_PARAM;
        a->f1[f] = f1[f];
        a->f2[f] = f2[f];
    }
    a->scale = P->scale;
    a->y = P->y;
    a->target = P->target;
    a->L = P->lv[0];
    return LC3D_OK;
}

int lc3d_predictor_predict(lc3d_predictor* P, const double* const* f1, const double* const* f2,
                           double* const* pred, void* stream) {
    if (!P || !f1 || !f2 || !pred) return LC3D_ERR_PARAM;
    OutArgs a{};
    LC3D_TRY(out_args(P, &a, f1, f2, true));
    for (int f = 0; f < 6; ++f) {
        if (!pred[f]) return LC3D_ERR_PARAM;
        a.pred[f] = pred[f];
    }
    PredDevice g(P->device);
    unpack_kernel<<<blocks_for((long long)P->N * P->N, 256), 256, 0, St(stream)>>>(a);
    LC3D_CUDA_TRY(cudaGetLastError());
    return LC3D_OK;
}

int lc3d_predictor_set_target(lc3d_predictor* P, const double* const* first, const double* const* f1,
                              const double* const* f2, void* stream) {
    if (!P || !first || !f1 || !f2) return LC3D_ERR_PARAM;
    OutArgs a{};
    LC3D_TRY(out_args(P, &a, f1, f2, false));
    for (int k = 0; k < 5; ++k) {
        if (!first[net_field(k)]) return LC3D_ERR_PARAM;
        a.first[net_field(k)] = first[net_field(k)];
    }
    PredDevice g(P->device);
    target_kernel<<<blocks_for(P->lv[0].NP, 128), 128, 0, St(stream)>>>(a);
    LC3D_CUDA_TRY(cudaGetLastError());
    return LC3D_OK;
}

int lc3d_predictor_backward(lc3d_predictor* P, float* loss, void* stream) {
    if (!P || !loss) return LC3D_ERR_PARAM;
    PredDevice g(P->device);
    return backward(P, loss, St(stream));
}

int lc3d_predictor_adam(lc3d_predictor* P, float lr, void* stream) {
    if (!P || !(lr > 0)) return LC3D_ERR_PARAM;
    PredDevice g(P->device);
    const float b1 = 0.9f, b2 = 0.999f;
    P->adam_t += 1;
    const float c1 = 1.0f - powf(b1, (float)P->adam_t), c2 = 1.0f - powf(b2, (float)P->adam_t);
    adam_kernel<<<blocks_for(P->np, 256), 256, 0, St(stream)>>>(P->params, P->grad, P->adam_m, P->adam_v, P->wbf,
                                                                P->np, lr, b1, b2, 1e-8f, c1, c2);
    LC3D_CUDA_TRY(cudaGetLastError());
    return LC3D_OK;
}

int lc3d_predictor_tensor(lc3d_predictor* P, int which, void** ptr, long long* bytes) {
    if (!P || !ptr || !bytes) return LC3D_ERR_PARAM;
    const long long n0 = P->lv[0].NP;
    switch (which) {
        case LC3D_PRED_INPUT: *ptr = P->x0; *bytes = n0 * 32 * 2; break;
        case LC3D_PRED_OUTPUT: *ptr = P->y; *bytes = n0 * 16 * 4; break;
        case LC3D_PRED_TARGET: *ptr = P->target; *bytes = n0 * 16 * 4; break;
        default: return LC3D_ERR_PARAM;
    }
    return LC3D_OK;
}

int lc3d_predictor_check_error(lc3d_predictor* P, void* stream) {
    if (!P) return LC3D_ERR_PARAM;
    PredDevice g(P->device);
    unsigned h = 0;
    LC3D_CUDA_TRY(cudaMemcpyAsync(&h, P->err, sizeof(unsigned), cudaMemcpyDeviceToHost, St(stream)));
    LC3D_CUDA_TRY(cudaStreamSynchronize(St(stream)));
    if (h) {
        LC3D_CUDA_TRY(cudaMemsetAsync(P->err, 0, sizeof(unsigned), St(stream)));
        return LC3D_ERR_TIMEOUT;
    }
    return LC3D_OK;
}

}  // extern "C"
