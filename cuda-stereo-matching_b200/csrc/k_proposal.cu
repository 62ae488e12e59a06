// Learned support-point proposal: feature pooling, the training kernels
// (fp32 forward / backward of the 4-layer 3x3 CNN, correlation loss, Adam)
// and the bf16 inference path (tcgen05 implicit-GEMM convolutions, top-4
// bins per candidate).  The reference has no learned component; the
// network, its parameter layout and the proposal rule are defined once, in
// the CPU oracle's module docstring, and restated here.
//
// Layouts.  Feature maps are NHWC: [image][Hd][Wd][32], image = 2*pair +
// view (0 left, 1 right).  Training parameters, per layer: W[tap][ci][co]
// (tap = 3*(dy+1) + (dx+1)) then b[co], fp32.  Inference weights: bf16
// B operands [layer][tap][co][ci] (K-major, 64-byte rows) plus fp32 bias.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstdint>
#include <initializer_list>
#include <type_traits>

#include "common.cuh"
#include "launch.cuh"
#include "proposal.h"

namespace elas {
namespace pn {

namespace {

// ---------------------------------------------------------------------------
// Pooled descriptor features: cell (x, y) of image v covers pixels
// [4x, 4x+4) x [4y, 4y+4).  Channel c < 16: (mean_c - 128) / 64; channel
// 16 + c: mean |byte_c - 128| / 64.  Both are exact in fp32 before the bf16
// rounding.
__global__ void k_features(const uint4* __restrict__ desc0, const uint4* __restrict__ desc1,
                           __nv_bfloat16* __restrict__ out, int W, int Hd, int Wd) {
    grid_dep_wait();
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y, v = blockIdx.z;
    if (x >= Wd) return;
    const uint4* D = v ? desc1 : desc0;
    int sum[16], dev[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) sum[c] = dev[c] = 0;
    for (int r = 0; r < 4; ++r)
        for (int q = 0; q < 4; ++q) {
            uint4 d = D[size_t(4 * y + r) * W + 4 * x + q];
            const uint32_t w4[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    int b = int((w4[k] >> (8 * j)) & 0xffu);
                    sum[4 * k + j] += b;
                    dev[4 * k + j] += abs(b - 128);
                }
        }
    __align__(16) __nv_bfloat16 o[CH];
#pragma unroll
    for (int c = 0; c < 16; ++c) {
        o[c] = __float2bfloat16_rn((float(sum[c]) * 0.0625f - 128.0f) * 0.015625f);
        o[16 + c] = __float2bfloat16_rn(float(dev[c]) * (1.0f / 1024.0f));
    }
    uint4* dst = reinterpret_cast<uint4*>(out + ((size_t(v) * Hd + y) * Wd + x) * CH);
    const uint4* src = reinterpret_cast<const uint4*>(o);
#pragma unroll
    for (int k = 0; k < 4; ++k) dst[k] = src[k];
}

__global__ void k_bf16_to_f32(const __nv_bfloat16* __restrict__ in, float* __restrict__ out, size_t n) {
    grid_dep_wait();
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
        out[i] = __bfloat162float(in[i]);
}

// ---------------------------------------------------------------------------
// Training convolution (fp32).  Bound by the FP32 pipes (9216 FMAs a cell),
// so two of them go in one instruction (twice 32 bits, rounded as two
// separate ones) and their operands stay in registers: a thread computes 16
// cells x 4 output channels, as eight pairs of cells eight rows apart, and
// loads 16 + 4 words from shared memory per input channel for 64 FMAs (8
// cells x 4 channels, one FMA an instruction: 12 words for 32 FMAs, 440 us a
// layer; 16 x 8, half as many warps: 457).  A group of 256 threads takes a
// 16 x 32 cell tile, held in shared memory with the two rows of a pair side
// by side, so that a pair's values arrive in one register pair at every tap;
// CT_PITCH values a cell let the cells of a warp read distinct banks.  One
// CTA per SM holds the weights and two such groups, each with a tile and a
// barrier of its own: one computes while the other stages.  Sums run over
// taps, then input channels, in order, as one chain per output.  `mask`
// (nullable) multiplies each input value by (mask > 0): the ReLU derivative
// when this kernel computes the gradient of the layer input.
// 32 images of 93 x 310 cells: 1726 us -> 361 us a layer (the FMAs alone: 252).
constexpr int CT_H = 16, CT_W = 32, CT_PITCH = CH + 2, CT_GROUP = 256, CT_GROUPS = 2;
constexpr int CT_THREADS = CT_GROUP * CT_GROUPS, CT_PAIRS = CT_H / 2 + 2;      // row pairs with the halo
constexpr int CT_TILE = CT_PAIRS * (CT_W + 2) * CT_PITCH;                       // float2 of one tile
constexpr size_t CONV_F32_SMEM = sizeof(float) * (TAPS * CH * CH + CT_GROUPS * CT_TILE * 2);
static_assert(CT_GROUP / 32 == CT_H / 2 && CT_W == 32 && CH == 32, "a warp per row pair");

// Four channels of one cell; vec: the base is 16-byte aligned.
__device__ __forceinline__ float4 load4(const float* p, bool vec) {
    return vec ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
}
__device__ __forceinline__ float4 masked4(float4 v, float4 m) {
    return make_float4(m.x > 0.0f ? v.x : 0.0f, m.y > 0.0f ? v.y : 0.0f, m.z > 0.0f ? v.z : 0.0f,
                       m.w > 0.0f ? v.w : 0.0f);
}

// Two FP32 values in a register pair: one instruction multiplies and adds both.
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ void fma2(uint64_t& acc, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

__device__ __forceinline__ void group_sync(int group) {
    asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(CT_GROUP) : "memory");
}

__global__ void __launch_bounds__(CT_THREADS, 1) k_conv_f32(const float* __restrict__ x,
                                                            const float* __restrict__ mask,
                                                            const float* __restrict__ w, const float* __restrict__ b,
                                                            float* __restrict__ y, int nimg, int Hd, int Wd, int relu,
                                                            int vec) {
    grid_dep_wait();
    extern __shared__ __align__(16) float conv_sm[];
    float* sw = conv_sm;                        // [TAPS][ci][co]
    const int group = threadIdx.x / CT_GROUP, tid = threadIdx.x % CT_GROUP;
    // [CT_PAIRS][CT_W + 2][CT_PITCH]
    float2* sx = reinterpret_cast<float2*>(conv_sm + TAPS * CH * CH) + group * CT_TILE;
    const int cog = tid & 7, cg = (tid >> 3) & 3, rp = tid >> 5;
    for (int i = threadIdx.x; i < TAPS * CH * CH; i += CT_THREADS) sw[i] = w[i];
    __syncthreads();
    const int tx = (Wd + CT_W - 1) / CT_W, ty = (Hd + CT_H - 1) / CT_H;
    const long long ntiles = (long long)nimg * tx * ty;
    for (long long tile = blockIdx.x + (long long)group * gridDim.x; tile < ntiles;
         tile += CT_GROUPS * (long long)gridDim.x) {
        const int n = int(tile / (tx * ty)), q = int(tile % (tx * ty));
        const int r0 = q / tx * CT_H, c0 = q % tx * CT_W;
        group_sync(group);              // the tile before has been read
        {
            const int k = tid % (CH / 4);
            int r = 0, j = tid / (CH / 4);
            const auto word = [&](int yy, int xx) {
                float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (yy >= 0 && yy < Hd && xx >= 0 && xx < Wd) {
                    const size_t at = ((size_t(n) * Hd + yy) * Wd + xx) * CH + 4 * k;
                    v = load4(x + at, vec);
                    if (mask) v = masked4(v, load4(mask + at, vec));
                }
                return v;
            };
#pragma unroll 4
            for (int i = tid; i < CT_PAIRS * (CT_W + 2) * (CH / 4); i += CT_GROUP) {
                const int yy = r0 + r - 1, xx = c0 + j - 1;
                const float4 lo = word(yy, xx), hi = word(yy + CT_H / 2, xx);
                float4* o = reinterpret_cast<float4*>(sx + (r * (CT_W + 2) + j) * CT_PITCH + 4 * k);
                o[0] = make_float4(lo.x, hi.x, lo.y, hi.y);
                o[1] = make_float4(lo.z, hi.z, lo.w, hi.w);
                j += CT_GROUP / (CH / 4);
                if (j >= CT_W + 2) { j -= CT_W + 2; ++r; }
            }
        }
        group_sync(group);
        // row pair rp, columns cg, cg + 4, ..., channels 4 cog ..
        uint64_t acc[8][4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const float bc = b ? b[4 * cog + c] : 0.0f;
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[i][c] = pack2(bc, bc);
        }
#pragma unroll 1
        for (int t = 0; t < TAPS; ++t) {
            const float2* xs = sx + ((rp + t / 3) * (CT_W + 2) + cg + t % 3) * CT_PITCH;
            const float* ws = sw + t * CH * CH + 4 * cog;
// unrolled in full: short loops moved registers about (421 in place of 361 us)
#pragma unroll
            for (int ci = 0; ci < CH; ci += 2) {
                ulonglong2 xv[8];
                float4 wv[2];
#pragma unroll
                for (int k = 0; k < 2; ++k) wv[k] = *reinterpret_cast<const float4*>(ws + (ci + k) * CH);
#pragma unroll
                for (int i = 0; i < 8; ++i) xv[i] = *reinterpret_cast<const ulonglong2*>(xs + 4 * i * CT_PITCH + ci);
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const uint64_t w2[4] = {pack2(wv[k].x, wv[k].x), pack2(wv[k].y, wv[k].y),
                                            pack2(wv[k].z, wv[k].z), pack2(wv[k].w, wv[k].w)};
#pragma unroll
                    for (int c = 0; c < 4; ++c)
#pragma unroll
                        for (int i = 0; i < 8; ++i) fma2(acc[i][c], k ? xv[i].y : xv[i].x, w2[c]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int xo = c0 + cg + 4 * i;
            if (xo >= Wd) continue;
            float2 v[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                v[c] = unpack2(acc[i][c]);
                if (relu) v[c] = make_float2(fmaxf(v[c].x, 0.0f), fmaxf(v[c].y, 0.0f));
            }
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int yy = r0 + rp + half * (CT_H / 2);
                if (yy >= Hd) continue;
                float* o = y + ((size_t(n) * Hd + yy) * Wd + xo) * CH + 4 * cog;
                const float4 q4 = half ? make_float4(v[0].y, v[1].y, v[2].y, v[3].y)
                                       : make_float4(v[0].x, v[1].x, v[2].x, v[3].x);
                if (vec) {
                    *reinterpret_cast<float4*>(o) = q4;
                } else {
                    o[0] = q4.x;
                    o[1] = q4.y;
                    o[2] = q4.z;
                    o[3] = q4.w;
                }
            }
        }
    }
}

// The same convolution, the same sums in the same order, for small maps: a
// block takes ROW_SEG cells of one image row x 32 output channels (lane =
// output channel, warp = cell), with the three input rows of the segment (and
// a one-cell halo) and all weights in shared memory.  A thread has one
// output, so a map of a few thousand cells still spreads over every SM,
// where k_conv_f32's tiles would leave most of them idle and one group would
// take 31-33 us for the first of them.
constexpr int ROW_SEG = 32;
constexpr size_t CONV_ROWS_SMEM = sizeof(float) * (TAPS * CH * CH + 3 * (ROW_SEG + 2) * CH);

__global__ void __launch_bounds__(ROW_SEG * CH) k_conv_f32_rows(const float* __restrict__ x,
                                                                const float* __restrict__ mask,
                                                                const float* __restrict__ w,
                                                                const float* __restrict__ b, float* __restrict__ y,
                                                                int Hd, int Wd, int relu) {
    grid_dep_wait();
    extern __shared__ float row_sm[];
    float* sw = row_sm;                                                   // [TAPS][ci][co]
    float(*sx)[ROW_SEG + 2][CH] = reinterpret_cast<float(*)[ROW_SEG + 2][CH]>(row_sm + TAPS * CH * CH);
    const int n = blockIdx.z, row = blockIdx.y, x0 = blockIdx.x * ROW_SEG;
    const int co = threadIdx.x & 31, cell = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < TAPS * CH * CH; i += blockDim.x) sw[i] = w[i];
    for (int i = threadIdx.x; i < 3 * (ROW_SEG + 2) * CH; i += blockDim.x) {
        const int c = i % CH, j = (i / CH) % (ROW_SEG + 2), r = i / (CH * (ROW_SEG + 2));
        const int yy = row + r - 1, xx = x0 + j - 1;
        float v = 0.0f;
        if (yy >= 0 && yy < Hd && xx >= 0 && xx < Wd) {
            const size_t at = ((size_t(n) * Hd + yy) * Wd + xx) * CH + c;
            v = x[at];
            if (mask && !(mask[at] > 0.0f)) v = 0.0f;
        }
        sx[r][j][c] = v;
    }
    __syncthreads();
    const int xo = x0 + cell;
    if (xo >= Wd) return;
    float acc = b ? b[co] : 0.0f;
#pragma unroll
    for (int t = 0; t < TAPS; ++t) {
        const float* xs = sx[t / 3][cell + t % 3];
        const float* ws = sw + t * CH * CH + co;
#pragma unroll 8
        for (int ci = 0; ci < CH; ++ci) acc = fmaf(xs[ci], ws[ci * CH], acc);
    }
    if (relu) acc = fmaxf(acc, 0.0f);
    y[((size_t(n) * Hd + row) * Wd + xo) * CH + co] = acc;
}

// Wt[8 - t][co][ci] = W[t][ci][co]: the gradient of a layer input is the
// same convolution of the output gradient with these weights.
__global__ void k_flip_weights(const float* __restrict__ w, float* __restrict__ wt) {
    grid_dep_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= TAPS * CH * CH) return;
    const int t = i / (CH * CH), ci = (i / CH) % CH, co = i % CH;
    wt[((TAPS - 1 - t) * CH + co) * CH + ci] = w[i];
}

// Weight and bias gradients: dW[t][ci][co] += sum_cells x[cell + off_t][ci] * g[cell][co],
// db[co] += sum g[cell][co], with g = dy * (y > 0) when `y` is given.  Bound
// by the FP32 pipes like the convolution, two FMAs an instruction: 64 threads hold all 9 x 32 x 32
// sums in registers (4 ci x 4 co x 9 taps each) and walk along a row of
// cells; a step loads the three new input words of the 3 x 3 window and one
// gradient word, 16 bytes each and a step ahead, for 144 FMAs.  A CTA runs four such groups,
// one per row of a 4 x 32 cell tile; the next tile arrives by cp.async
// meanwhile (the registers leave room for one CTA per SM, so nothing else
// would cover its latency).  CTAs are persistent: the four groups' sums are
// added in shared memory once, at the end, so dW receives one atomic per
// weight and CTA (a CTA per 8-row band used to add 26 times as many).
// 32 images of 93 x 310 cells: 964 us -> 370 us a layer (one FMA an
// instruction and a division per staged word: 441).
constexpr int WG_H = 4, WG_W = 32, WG_THREADS = 256;
constexpr int WG_X = (WG_H + 2) * (WG_W + 2) * CH, WG_G = WG_H * WG_W * CH;      // floats of the two tiles
constexpr int WG_SUMS = TAPS * CH * CH + CH;
constexpr int WG_BUF = WG_X + 2 * WG_G;      // inputs, output gradients and, with a mask, outputs of one tile
constexpr size_t WGRAD_SMEM = sizeof(float) * 2 * WG_BUF;
static_assert(WG_SUMS <= 2 * WG_BUF, "the final sums reuse the tiles");

// 16 bytes global -> shared in the background (zeros where !ok).
__device__ __forceinline__ void copy4_async(float* dst, const float* src, bool ok, bool vec) {
    const uint32_t d = smem_u32(dst);
    if (vec) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(ok ? 16 : 0) : "memory");
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d + 4 * k), "l"(src + k),
                         "r"(ok ? 4 : 0)
                         : "memory");
    }
}

__global__ void __launch_bounds__(WG_THREADS, 1) k_conv_wgrad(const float* __restrict__ x,
                                                              const float* __restrict__ dy,
                                                              const float* __restrict__ y, float* __restrict__ dw,
                                                              float* __restrict__ db, int nimg, int Hd, int Wd,
                                                              int vec) {
    grid_dep_wait();
    extern __shared__ __align__(16) float wg_sm[];
    const int tid = threadIdx.x, cog = tid & 7, cig = (tid >> 3) & 7, row = tid >> 6;
    uint64_t acc[TAPS][2][4];           // [tap][ci pair][co]
    float bacc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int t = 0; t < TAPS; ++t)
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[t][i][c] = 0;
    const int tx = (Wd + WG_W - 1) / WG_W, ty = (Hd + WG_H - 1) / WG_H;
    const long long ntiles = (long long)nimg * tx * ty;
    // tile buffer: inputs [WG_H + 2][WG_W + 2][CH], then dy and y [WG_H][WG_W][CH]
    auto stage = [&](long long tile, float* buf) {
        const int n = int(tile / (tx * ty)), q = int(tile % (tx * ty));
        const int r0 = q / tx * WG_H, c0 = q % tx * WG_W;
        // a word of 32 columns' 8 per thread, row by row; the two last columns' words by 96 threads
        const int k = tid % (CH / 4), j = tid / (CH / 4);
        const auto copy_x = [&](int r, int col) {
            const int yy = r0 + r - 1, xx = c0 + col - 1;
            const bool ok = yy >= 0 && yy < Hd && xx >= 0 && xx < Wd;
            copy4_async(buf + (r * (WG_W + 2) + col) * CH + 4 * k,
                        ok ? x + ((size_t(n) * Hd + yy) * Wd + xx) * CH + 4 * k : x, ok, vec);
        };
#pragma unroll
        for (int r = 0; r < WG_H + 2; ++r) copy_x(r, j);
        if (j < 2 * (WG_H + 2)) copy_x(j >> 1, WG_W + (j & 1));
#pragma unroll
        for (int r = 0; r < WG_H; ++r) {
            const bool ok = r0 + r < Hd && c0 + j < Wd;
            const size_t at = ok ? ((size_t(n) * Hd + r0 + r) * Wd + c0 + j) * CH + 4 * k : 0;
            float* g = buf + WG_X + (r * WG_W + j) * CH + 4 * k;
            copy4_async(g, dy + at, ok, vec);
            if (y) copy4_async(g + WG_G, y + at, ok, vec);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int cur = 0;
    if (blockIdx.x < ntiles) stage(blockIdx.x, wg_sm);
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x, cur ^= 1) {
        if (tile + gridDim.x < ntiles) {
            stage(tile + gridDim.x, wg_sm + (cur ^ 1) * WG_BUF);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const float* sx = wg_sm + cur * WG_BUF;
        const float* sg = sx + WG_X;
        const float* xr = sx + row * (WG_W + 2) * CH + 4 * cig;
        const float* gr = sg + row * WG_W * CH + 4 * cog;
        // columns j .. j + 2 of the window and j + 3, on its way; column c lies in win[.][c % 4]
        float4 win[3][4];
        const auto load_g = [&](int j) {
            const float4 g = *reinterpret_cast<const float4*>(gr + j * CH);
            return y ? masked4(g, *reinterpret_cast<const float4*>(gr + WG_G + j * CH)) : g;
        };
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c)
                win[r][c] = *reinterpret_cast<const float4*>(xr + (r * (WG_W + 2) + c) * CH);
        float4 g_next = load_g(0);
#pragma unroll 2
        for (int j0 = 0; j0 < WG_W; j0 += 4)
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                const int j = j0 + p;
                const float4 g = g_next;
                const uint64_t g2[4] = {pack2(g.x, g.x), pack2(g.y, g.y), pack2(g.z, g.z), pack2(g.w, g.w)};
                // (past the row's end: a word of the next row, not used)
#pragma unroll
                for (int r = 0; r < 3; ++r)
                    win[r][(p + 3) & 3] = *reinterpret_cast<const float4*>(xr + (r * (WG_W + 2) + j + 3) * CH);
                g_next = load_g(min(j + 1, WG_W - 1));
#pragma unroll
                for (int r = 0; r < 3; ++r)
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const float4 v = win[r][(p + c) & 3];
                        const uint64_t v01 = pack2(v.x, v.y), v23 = pack2(v.z, v.w);
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            fma2(acc[3 * r + c][0][k], v01, g2[k]);
                            fma2(acc[3 * r + c][1][k], v23, g2[k]);
                        }
                    }
                if (cig == 0) {
                    bacc[0] += g.x;
                    bacc[1] += g.y;
                    bacc[2] += g.z;
                    bacc[3] += g.w;
                }
            }
        __syncthreads();                // the buffer is free for the tile after next
    }
    // the four groups' sums, group by group, into shared memory, then one atomic per weight
    for (int g = 0; g < WG_H; ++g) {
        __syncthreads();
        if (row != g) continue;
#pragma unroll
        for (int t = 0; t < TAPS; ++t)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float4* o = reinterpret_cast<float4*>(wg_sm + (t * CH + 4 * cig + i) * CH + 4 * cog);
                float v4[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float2 pr = unpack2(acc[t][i >> 1][c]);
                    v4[c] = i & 1 ? pr.y : pr.x;
                }
                float4 v = make_float4(v4[0], v4[1], v4[2], v4[3]);
                if (g) {
                    const float4 p = *o;
                    v = make_float4(p.x + v.x, p.y + v.y, p.z + v.z, p.w + v.w);
                }
                *o = v;
            }
        if (cig == 0)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                float* o = wg_sm + TAPS * CH * CH + 4 * cog + c;
                *o = g ? *o + bacc[c] : bacc[c];
            }
    }
    __syncthreads();
    for (int i = tid; i < TAPS * CH * CH; i += WG_THREADS) atomicAdd(&dw[i], wg_sm[i]);
    if (tid < CH) atomicAdd(&db[tid], wg_sm[TAPS * CH * CH + tid]);
}
static_assert(WG_W * (CH / 4) == WG_THREADS, "a thread stages one word of each row");
static_assert(WG_W % 4 == 0, "four cells a turn of the window's columns");

// Correlation scores, softmax cross-entropy and the feature gradients, one
// warp per label (pair, cx, cy, bin) in turn.  Bound by the L2 atomics of
// the gradient (64 bins x 32 channels a label).  Eight lanes share a bin,
// four channels each, so features are read and gradients added 16 bytes a
// lane, four bins an access; the partial scores of a lane's 16 bins are
// then reduced together, each exchange halving the bins it still holds.
// Lane l ends with the scores of bins 4 (2 (l & 7) + k) + (l >> 3), k = 0, 1.
// A warp keeps its labels' loss in 64 bits and a CTA adds it once, so the
// sum over some 10^4 labels rounds a few hundred times instead of once a
// label.  32000 labels of 16 pairs of 93 x 310 cells: 220 us -> 86 us.
constexpr int CORR_THREADS = 256, CORR_CTAS_PER_SM = 4;
__global__ void __launch_bounds__(CORR_THREADS, CORR_CTAS_PER_SM)
    k_corr_loss(const float* __restrict__ F, const int32_t* __restrict__ labels, int nlab, int Hd, int Wd, int D,
                float inv_n, float* __restrict__ dF, float* __restrict__ loss_sum, int32_t* __restrict__ correct,
                int vec) {
    grid_dep_wait();
    __shared__ double wl[CORR_THREADS / 32];
    __shared__ int wh[CORR_THREADS / 32];
    const int lane = threadIdx.x & 31, w = bin_width(D);
    const int grp = lane >> 3, c4 = 4 * (lane & 7);        // the lane's bins modulo 4 and its channels
    double loss = 0.0;
    int hits = 0;
    auto add4 = [&](float* p, float4 v) {
        if (vec) {
            atomicAdd(reinterpret_cast<float4*>(p), v);
        } else {
            atomicAdd(p, v.x);
            atomicAdd(p + 1, v.y);
            atomicAdd(p + 2, v.z);
            atomicAdd(p + 3, v.w);
        }
    };
    for (int lab = (blockIdx.x * CORR_THREADS + threadIdx.x) >> 5; lab < nlab;
         lab += gridDim.x * (CORR_THREADS / 32)) {
        const int pair = labels[4 * lab], cx = labels[4 * lab + 1], cy = labels[4 * lab + 2], tb = labels[4 * lab + 3];
        if (cx - bin_shift(tb, w) < 0) continue;           // the oracle skips these labels
        const size_t Lrow = ((size_t(2 * pair) * Hd + cy) * Wd) * CH;
        const size_t Rrow = ((size_t(2 * pair + 1) * Hd + cy) * Wd) * CH;
        const float4 fl = load4(F + Lrow + size_t(cx) * CH + c4, vec);
        const float* fr = F + Rrow + c4;
        float p[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int x2 = cx - bin_shift(4 * i + grp, w);
            p[i] = 0.0f;
            if (x2 >= 0) {
                const float4 v = load4(fr + x2 * CH, vec);
                p[i] = fmaf(fl.x, v.x, fl.y * v.y) + fmaf(fl.z, v.z, fl.w * v.w);
            }
        }
#pragma unroll
        for (int o = 4, n = 8; o > 0; o >>= 1, n >>= 1) {
            const bool up = (lane & o) != 0;
#pragma unroll
            for (int i = 0; i < n; ++i) {
                const float keep = up ? p[i + n] : p[i], give = up ? p[i] : p[i + n];
                p[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
        }
        float s[2];
        int bin[2];
        bool valid[2];
        float m = -INFINITY;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            s[k] = SCALE * p[k];
            bin[k] = 4 * (2 * (lane & 7) + k) + grp;
            valid[k] = cx - bin_shift(bin[k], w) >= 0;
            if (valid[k]) m = fmaxf(m, s[k]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        float e[2], z = 0.0f;
#pragma unroll
        for (int k = 0; k < 2; ++k) { e[k] = valid[k] ? expf(s[k] - m) : 0.0f; z += e[k]; }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
        // argmax (lowest bin on ties) for the accuracy count
        float best = -INFINITY;
        int bi = NBINS;
#pragma unroll
        for (int k = 0; k < 2; ++k)
            if (valid[k] && (s[k] > best)) { best = s[k]; bi = bin[k]; }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
        }
        const float st = __shfl_sync(0xffffffffu, (tb >> 2) & 1 ? s[1] : s[0], 8 * (tb & 3) + (tb >> 3));
        loss -= double(st - m - logf(z));
        hits += bi == tb ? 1 : 0;
        float g[2];
#pragma unroll
        for (int k = 0; k < 2; ++k)
            g[k] = valid[k] ? (e[k] / z - (bin[k] == tb ? 1.0f : 0.0f)) * inv_n * SCALE : 0.0f;
        // dF_L[c] = sum_b g_b F_R(x - s_b)[c];  dF_R(x - s_b)[c] += g_b F_L[c]
        float4 dl = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        float* dr = dF + Rrow + c4;
#pragma unroll 4
        for (int i = 0; i < 16; ++i) {
            const float gb = __shfl_sync(0xffffffffu, i & 1 ? g[1] : g[0], (lane & 24) | (i >> 1));
            const int x2 = cx - bin_shift(4 * i + grp, w);
            if (x2 < 0 || gb == 0.0f) continue;
            const float4 v = load4(fr + x2 * CH, vec);
            dl = make_float4(fmaf(gb, v.x, dl.x), fmaf(gb, v.y, dl.y), fmaf(gb, v.z, dl.z), fmaf(gb, v.w, dl.w));
            add4(dr + x2 * CH, make_float4(gb * fl.x, gb * fl.y, gb * fl.z, gb * fl.w));
        }
        __syncwarp();
#pragma unroll
        for (int o = 8; o < 32; o <<= 1) {
            dl.x += __shfl_xor_sync(0xffffffffu, dl.x, o);
            dl.y += __shfl_xor_sync(0xffffffffu, dl.y, o);
            dl.z += __shfl_xor_sync(0xffffffffu, dl.z, o);
            dl.w += __shfl_xor_sync(0xffffffffu, dl.w, o);
        }
        if (grp == 0) add4(dF + Lrow + size_t(cx) * CH + c4, dl);
    }
    if (lane == 0) {
        wl[threadIdx.x >> 5] = loss;
        wh[threadIdx.x >> 5] = hits;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < CORR_THREADS / 32; ++k) {
            loss += wl[k];
            hits += wh[k];
        }
        atomicAdd(loss_sum, float(loss));
        if (hits) atomicAdd(correct, hits);
    }
}

__global__ void k_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, int n, float lr, float b1, float b2, float eps, float c1, float c2) {
    grid_dep_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

}  // namespace

cudaError_t launch_features(const uint4* desc0, const uint4* desc1, __nv_bfloat16* out, int W, int H,
                            cudaStream_t st) {
    const int Hd = H / 4, Wd = W / 4;
    if (Hd <= 0 || Wd <= 0) return cudaSuccess;
    launch_k(k_features, dim3((Wd + 63) / 64, Hd, 2), 64, 0, st, desc0, desc1, out, W, Hd, Wd);
    return cudaGetLastError();
}

cudaError_t launch_bf16_to_f32(const __nv_bfloat16* in, float* out, size_t n, cudaStream_t st) {
    k_bf16_to_f32<<<1024, 256, 0, st>>>(in, out, n);
    return cudaGetLastError();
}

namespace {
// Whether every given pointer (null: none) allows 16-byte accesses; the
// training kernels fall back to 4-byte ones where a caller's do not.
bool aligned16(std::initializer_list<const void*> ps) {
    uintptr_t m = 0;
    for (const void* p : ps) m |= reinterpret_cast<uintptr_t>(p);
    return (m & 15) == 0;
}
int sm_count() {
    int dev = 0, n = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n;
}
int tile_grid(long long tiles, int ctas) { return int(tiles < ctas ? tiles : ctas); }
}  // namespace

cudaError_t launch_conv_f32(const float* x, const float* mask, const float* w, const float* b, float* y, int nimg,
                            int Hd, int Wd, int relu, cudaStream_t st) {
    const int sms = sm_count();
    // 83 cells an SM (12284): rows of 1 x 16 x 32, 2 x 60 x 80 and 10 x 20 x
    // 64 cells take 13, 29 and 29 us, tiles 33 of all three; 2 x 93 x 80
    // (14880 cells) 39 and 33, 2 x 93 x 310 115 and 33
    if ((long long)nimg * Hd * Wd <= 83LL * sms) {
        allow_smem(k_conv_f32_rows);
        k_conv_f32_rows<<<dim3((Wd + ROW_SEG - 1) / ROW_SEG, Hd, nimg), ROW_SEG * CH, CONV_ROWS_SMEM, st>>>(
            x, mask, w, b, y, Hd, Wd, relu);
        return cudaGetLastError();
    }
    allow_smem(k_conv_f32);
    const long long tiles = (long long)nimg * ((Wd + CT_W - 1) / CT_W) * ((Hd + CT_H - 1) / CT_H);
    k_conv_f32<<<tile_grid(tiles, sms), CT_THREADS, CONV_F32_SMEM, st>>>(x, mask, w, b, y, nimg, Hd, Wd, relu,
                                                                         aligned16({x, mask, y}));
    return cudaGetLastError();
}

cudaError_t launch_flip_weights(const float* w, float* wt, cudaStream_t st) {
    k_flip_weights<<<(TAPS * CH * CH + 255) / 256, 256, 0, st>>>(w, wt);
    return cudaGetLastError();
}

cudaError_t launch_conv_wgrad(const float* x, const float* dy, const float* y, float* dw, float* db, int nimg,
                              int Hd, int Wd, cudaStream_t st) {
    allow_smem(k_conv_wgrad);
    const long long tiles = (long long)nimg * ((Wd + WG_W - 1) / WG_W) * ((Hd + WG_H - 1) / WG_H);
    k_conv_wgrad<<<tile_grid(tiles, sm_count()), WG_THREADS, WGRAD_SMEM, st>>>(x, dy, y, dw, db, nimg, Hd, Wd,
                                                                               aligned16({x, dy, y}));
    return cudaGetLastError();
}

cudaError_t launch_corr_loss(const float* F, const int32_t* labels, int nlab, int Hd, int Wd, int D, float* dF,
                             float* loss_sum, int32_t* correct, cudaStream_t st) {
    if (nlab <= 0) return cudaSuccess;
    const int ctas = tile_grid((nlab + CORR_THREADS / 32 - 1) / (CORR_THREADS / 32), CORR_CTAS_PER_SM * sm_count());
    k_corr_loss<<<ctas, CORR_THREADS, 0, st>>>(F, labels, nlab, Hd, Wd, D, 1.0f / float(nlab), dF,
                                                         loss_sum, correct, aligned16({F, dF}));
    return cudaGetLastError();
}

cudaError_t launch_adam(float* p, const float* g, float* m, float* v, int n, float lr, float b1, float b2, float eps,
                        int t, cudaStream_t st) {
    const float c1 = 1.0f - powf(b1, float(t)), c2 = 1.0f - powf(b2, float(t));
    k_adam<<<(n + 255) / 256, 256, 0, st>>>(p, g, m, v, n, lr, b1, b2, eps, c1, c2);
    return cudaGetLastError();
}

}  // namespace pn
}  // namespace elas
