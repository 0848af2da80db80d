// FP32 convolutions of the network's training step (forward with stored activations, gradients
// for the inputs and for the weights), on the CUDA cores: every product and sum is one FP32 FMA.
//
// A training step at 32 crops of 96 x 96 is 17 G multiply-adds, 0.46 ms at the FP32 rate (37.4 T
// FMA/s measured), against 0.1 ms of HBM traffic: the FMA pipe bounds it, so the kernels are tiled
// to keep it fed. A block stages a 16 x 16 pixel tile with its halo in shared memory and each
// thread accumulates an outer product in registers: 4 pixels x 8 channels (convolutions) or
// 3 taps x 4 input x 8 output channels (weight gradients), as pairs of channels in the packed
// FP32x2 FMA, which needs half the issue slots and rounds each lane as fmaf does. A 16-byte shared
// load then feeds 5 to 10 packed FMAs. One output's products are summed in a fixed order: bias, then
// taps, then channels, each ascending.
#pragma once

#include <cuda_bf16.h>

#include <algorithm>

#include "common.cuh"
#include "ffpair2.cuh"

namespace gfgpu {
namespace nn {

constexpr int kTrainTile = 16; // pixels per tile edge

__device__ __forceinline__ f2 f2_fma_acc(f2 a, f2 b, f2 c)
{
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

template <int BYTES>
__device__ __forceinline__ void cp_async_zfill(void* sdst, const void* gsrc, bool valid)
{
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(sdst));
    const int n = valid ? BYTES : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(s), "l"(gsrc), "n"(BYTES), "r"(n) : "memory");
}

__device__ __forceinline__ void cp_async_commit()
{
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// all but the latest `N` groups of this thread's copies have landed
template <int N>
__device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

struct TrainGrid {
    int B, H, W, tx, ty; // tx, ty: tiles per row and column of an image
    int64_t tiles;
};

inline TrainGrid train_grid(int B, int H, int W)
{
    TrainGrid g{B, H, W, (W + kTrainTile - 1) / kTrainTile, (H + kTrainTile - 1) / kTrainTile, 0};
    g.tiles = static_cast<int64_t>(B) * g.tx * g.ty;
    return g;
}

// Pixels (y0 - halo .. y0 + 15 + halo) x (x0 - halo ..) of image b of X [B, H, W, C] into `s`
// [16 + 2 halo][16 + 2 halo][C], zeros outside the image, as one group of asynchronous copies of
// min(16, 4 C) bytes where `vec` (X is aligned for them), else of one float. SWZ: the 8 chunks of 4
// channels of a pixel in column x are stored in the order chunk ^ (x & 7), so that a warp that
// reads one chunk of 8 neighbouring pixels meets 32 different banks without padding.
template <int C, bool SWZ>
__device__ __forceinline__ void stage_tile(const float* __restrict__ X, const TrainGrid& g, int64_t b, int y0,
                                           int x0, int halo, bool vec, float* s)
{
    const int hw = kTrainTile + 2 * halo;
    const float* img = X + b * g.H * g.W * C;
    constexpr int V = C >= 4 ? 4 : C; // floats per copy
    constexpr int N = C / V;          // copies per pixel
    const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    for (int r = threadIdx.x >> 5; r < hw; r += warps) {
        const int yy = y0 - halo + r;
        const bool iny = yy >= 0 && yy < g.H;
        const float* row = img + (static_cast<int64_t>(yy) * g.W + x0 - halo) * C;
        for (int i = lane; i < hw * N; i += 32) {
            const int x = i / N, c = (i - x * N) * V;
            const bool in = iny && x0 - halo + x >= 0 && x0 - halo + x < g.W;
            const float* src = in ? row + x * C + c : X;
            float* dst = s + (r * hw + x) * C + (SWZ ? (c ^ ((x & 7) * 4)) : c);
            if (vec) {
                cp_async_zfill<4 * V>(dst, src, in);
            }
            else {
#pragma unroll
                for (int k = 0; k < V; ++k) cp_async_zfill<4>(dst + k, in ? src + k : X, in);
            }
        }
    }
}

// image and first pixel of a tile
__device__ __forceinline__ void tile_origin(const TrainGrid& g, int64_t tile, int64_t& b, int& y0, int& x0)
{
    b = tile / (g.tx * g.ty);
    const int rem = static_cast<int>(tile - b * g.tx * g.ty), tyi = rem / g.tx;
    y0 = tyi * kTrainTile;
    x0 = (rem - tyi * g.tx) * kTrainTile;
}

inline int tile_floats(int C, int halo)
{
    const int hw = kTrainTile + 2 * halo;
    return hw * hw * C;
}

inline size_t conv_smem(int CI, int dil)
{
    return (static_cast<size_t>(9 * CI * 32) + tile_floats(CI, dil)) * sizeof(float);
}

// 3x3 convolution with CI input and 32 output channels.
//   BWD = false: Y = relu(b + sum_t sum_ci X[p + dil off_t, ci] W[t, ci, co]), W [9][CI][32];
//   BWD = true:  Y = (sum_t sum_co X[p - dil off_t, co] W[t, ci, co]) where act > 0, else 0:
//                the gradient for the input of a layer 32 -> CI, W [9][32][CI].
// 256 threads, 256 pixels x 32 channels: a thread has 8 output channels (cg) of 4 pixels (columns gl
// and gl + 8 of two rows). Per 4 input channels a thread issues 4 + 8 16-byte shared
// loads for 64 packed FMAs. Two blocks per SM (111 KB each at dilation 4, 128 registers): one
// computes while the other copies its tile, and four warps per scheduler cover the shared loads.
// 32 -> 32 at 32 x 96 x 96: 108 us forward, 122 us for the data gradient (72 us at the FMA rate);
// one block with two tiles in shared memory 118 / 141 us (two warps per scheduler); a pixel per
// thread, each weight read from shared memory for one FMA, 477 / 519 us. Shared-memory reads bound
// it: with 4 channel groups and 2 pixels in a quarter-warp 111 / 124 us. The gradient's ReLU mask is
// read as bits before the products (a step of 32 crops 861 -> 854 us against reads in the epilogue,
// one after the other). With 2 or 4 input channels there is little to compute per staged byte: three
// blocks per SM.
template <int CI, bool BWD>
__global__ void __launch_bounds__(256, CI == 32 ? 2 : 3)
k_conv_tile(const float* __restrict__ X, const __nv_bfloat16* __restrict__ W, const float* __restrict__ bias,
            int dil, TrainGrid g, const float* __restrict__ act, bool vec, float* __restrict__ Y)
{
    constexpr bool SWZ = CI == 32;
    extern __shared__ __align__(16) float sm[];
    const int hw = kTrainTile + 2 * dil;
    float* ws = sm;               // [9 CI][32]
    float* xs = sm + 9 * CI * 32; // [hw][hw][CI]
#pragma unroll 12
    for (int i = threadIdx.x; i < 9 * CI * 32; i += 256) {
        if constexpr (BWD) {
            // shared [t][co][ci] from global [t][ci = 32][co = CI]
            const int t = i / (32 * CI), r = i - t * 32 * CI, co = r / 32, ci = r - co * 32;
            ws[i] = __bfloat162float(W[(t * 32 + ci) * CI + co]);
        }
        else {
            ws[i] = __bfloat162float(W[i]);
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // a quarter-warp's 16-byte shared loads take 2 clocks for up to two different chunks, else 4: with 32
    // input channels it holds 2 groups of output channels and 4 pixels (the 8 weight loads are the cheap
    // ones), else 4 groups and 2 pixels
    const int cg = (SWZ ? (lane & 1) | ((lane >> 2) & 2) : lane & 3) * 8;
    const int gl = SWZ ? ((lane >> 1) & 3) | ((lane >> 2) & 4) : lane >> 2;
    const int sgn = BWD ? -dil : dil;
    f2 b0[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
        b0[k] = BWD ? f2_make(0.0f, 0.0f) : f2_make(__ldg(bias + cg + 2 * k), __ldg(bias + cg + 2 * k + 1));
    for (int64_t tile = blockIdx.x; tile < g.tiles; tile += gridDim.x) {
        int64_t b;
        int y0, x0;
        tile_origin(g, tile, b, y0, x0);
        stage_tile<CI, SWZ>(X, g, b, y0, x0, dil, vec, xs);
        cp_async_commit();
        // bit 8 j + k: the activation of pixel j and channel cg + k is positive, read while the copies land
        [[maybe_unused]] uint32_t pos = 0;
        if constexpr (BWD) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int yy = y0 + 2 * warp + (j >> 1), xx = x0 + gl + 8 * (j & 1);
                if (yy >= g.H || xx >= g.W) continue;
                const float* a = act + ((b * g.H + yy) * g.W + xx) * 32 + cg;
                const float4 m0 = *reinterpret_cast<const float4*>(a), m1 = *reinterpret_cast<const float4*>(a + 4);
                const float m[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
#pragma unroll
                for (int k = 0; k < 8; ++k) pos |= (m[k] > 0.0f ? 1u : 0u) << (8 * j + k);
            }
        }
        cp_async_wait<0>();
        __syncthreads();
        f2 acc[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[j][k] = b0[k];
#pragma unroll 1
        for (int t = 0; t < 9; ++t) {
            const int col = gl + dil + (t % 3 - 1) * sgn, row = 2 * warp + dil + (t / 3 - 1) * sgn;
            const float* xt = xs + (row * hw + col) * CI;
            const int key = SWZ ? (col & 7) * 4 : 0; // the same for columns col and col + 8
            const float* wt = ws + t * CI * 32 + cg;
            constexpr int V = CI >= 4 ? 4 : CI;
#pragma unroll
            for (int c0 = 0; c0 < CI; c0 += V) {
                float a[4][V];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float* p = xt + ((j >> 1) * hw + 8 * (j & 1)) * CI + (c0 ^ key);
                    if constexpr (V == 4) {
                        const float4 q = *reinterpret_cast<const float4*>(p);
                        a[j][0] = q.x;
                        a[j][1] = q.y;
                        a[j][2] = q.z;
                        a[j][3] = q.w;
                    }
                    else {
                        const float2 q = *reinterpret_cast<const float2*>(p);
                        a[j][0] = q.x;
                        a[j][1] = q.y;
                    }
                }
#pragma unroll
                for (int c = 0; c < V; ++c) {
                    const ulonglong2 w0 = *reinterpret_cast<const ulonglong2*>(wt + (c0 + c) * 32);
                    const ulonglong2 w1 = *reinterpret_cast<const ulonglong2*>(wt + (c0 + c) * 32 + 4);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const f2 x2 = f2_make(a[j][c], a[j][c]);
                        acc[j][0] = f2_fma_acc(x2, w0.x, acc[j][0]);
                        acc[j][1] = f2_fma_acc(x2, w0.y, acc[j][1]);
                        acc[j][2] = f2_fma_acc(x2, w1.x, acc[j][2]);
                        acc[j][3] = f2_fma_acc(x2, w1.y, acc[j][3]);
                    }
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int yy = y0 + 2 * warp + (j >> 1), xx = x0 + gl + 8 * (j & 1);
            if (yy >= g.H || xx >= g.W) continue;
            const int64_t o = ((b * g.H + yy) * g.W + xx) * 32 + cg;
            float v[8];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                v[2 * k] = f2_lo(acc[j][k]);
                v[2 * k + 1] = f2_hi(acc[j][k]);
            }
            if constexpr (BWD) {
#pragma unroll
                for (int k = 0; k < 8; ++k) v[k] = (pos >> (8 * j + k)) & 1u ? v[k] : 0.0f;
            }
            else {
#pragma unroll
                for (int k = 0; k < 8; ++k) v[k] = fmaxf(v[k], 0.0f);
            }
            *reinterpret_cast<float4*>(Y + o) = make_float4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<float4*>(Y + o + 4) = make_float4(v[4], v[5], v[6], v[7]);
        }
        __syncthreads(); // the tile is read before the next one is copied over it
    }
}

inline size_t conv_out_smem(int dil)
{
    return (static_cast<size_t>(9 * 32 * 2) + tile_floats(32, dil)) * sizeof(float);
}

// Output layer 32 -> 2: Y = b + sum_t sum_ci X[p + dil off_t, ci] W[t, ci, co]. Two pixels (of rows ly
// and ly + 8) of the staged tile per thread, a pixel's two outputs the lanes of one packed accumulator;
// 16-byte shared loads bound it (4 clocks for the pixels of a warp, 2 for each of two weights), so the
// weights serve two pixels. Five blocks per SM overlap their copies. 24 us at 32 x 96 x 96 (27 us with a
// pixel per thread; 300 us with a thread's pixel read from global memory one float at a time).
constexpr int kOutThreads = kTrainTile * kTrainTile / 2;

__global__ void __launch_bounds__(kOutThreads)
k_conv_out(const float* __restrict__ X, const __nv_bfloat16* __restrict__ W, const float* __restrict__ bias,
           int dil, TrainGrid g, float* __restrict__ Y)
{
    extern __shared__ __align__(16) float sm[];
    const int hw = kTrainTile + 2 * dil;
    float* ws = sm;              // [9][32][2]
    float* xs = sm + 9 * 32 * 2; // [hw][hw][32]
    for (int i = threadIdx.x; i < 9 * 32 * 2; i += kOutThreads) ws[i] = __bfloat162float(W[i]);
    const int ly = threadIdx.x / kTrainTile, lx = threadIdx.x % kTrainTile;
    for (int64_t tile = blockIdx.x; tile < g.tiles; tile += gridDim.x) {
        int64_t b;
        int y0, x0;
        tile_origin(g, tile, b, y0, x0);
        stage_tile<32, true>(X, g, b, y0, x0, dil, true, xs);
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
        f2 acc[2];
        acc[0] = acc[1] = f2_make(__ldg(bias), __ldg(bias + 1));
#pragma unroll
        for (int t = 0; t < 9; ++t) {
            const int col = lx + dil + dil * (t % 3 - 1), key = (col & 7) * 4;
            const float* p = xs + ((ly + dil + dil * (t / 3 - 1)) * hw + col) * 32;
#pragma unroll
            for (int c = 0; c < 32; c += 4) {
                const ulonglong2 w0 = *reinterpret_cast<const ulonglong2*>(ws + (t * 32 + c) * 2);
                const ulonglong2 w1 = *reinterpret_cast<const ulonglong2*>(ws + (t * 32 + c) * 2 + 4);
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const float4 q = *reinterpret_cast<const float4*>(p + j * (kTrainTile / 2) * hw * 32 + (c ^ key));
                    acc[j] = f2_fma_acc(f2_make(q.x, q.x), w0.x, acc[j]);
                    acc[j] = f2_fma_acc(f2_make(q.y, q.y), w0.y, acc[j]);
                    acc[j] = f2_fma_acc(f2_make(q.z, q.z), w1.x, acc[j]);
                    acc[j] = f2_fma_acc(f2_make(q.w, q.w), w1.y, acc[j]);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int yy = y0 + ly + j * (kTrainTile / 2);
            if (yy < g.H && x0 + lx < g.W) {
                const int64_t o = (b * g.H + yy) * g.W + x0 + lx;
                *reinterpret_cast<float2*>(Y + o * 2) = make_float2(f2_lo(acc[j]), f2_hi(acc[j]));
            }
        }
        __syncthreads();
    }
}

constexpr int kWgradThreads = 384; // 12 warps: 3 tap rows x 4 groups of 4 pixel rows

inline size_t wgrad_smem(int CI, int CO, int dil)
{
    const size_t tiles = 2 * (tile_floats(CI, dil) + tile_floats(CO, 0));
    const size_t sums = 4 * 9 * CI * CO + kWgradThreads;
    return std::max(tiles, sums) * sizeof(float);
}

// Weight gradient of a layer CI -> CO: per block, over its tiles (blockIdx, blockIdx + gridDim,
// ...), partial sums of dW[t, ci, co] = sum_p X[p + dil off_t, ci] dY[p, co] and db[co] =
// sum_p dY[p, co]; partial [gridDim.x][9 CI CO + CO]. A warp takes the three taps of one row over
// four pixel rows of the tile and keeps its sums in registers over all tiles; a lane owns 4 input
// channels and 8 (of 32) or both (of 2) output channels of each tap, and where that takes less
// than 32 lanes the rest of the lane index walks the pixels. At the end the pixel lanes' and the
// four row groups' sums are added in a fixed order. 32 -> 32: 5 shared loads of 16 bytes for 48
// packed FMAs; the next tile is copied while one is computed. 32 -> 32 at 32 x 96 x 96: 104 us (72
// us at the FMA rate), 4 -> 32 29 us, 32 -> 2 25 us; with a warp per tap (3 loads per 16 FMAs, nine
// warps that share four schedulers unevenly) and one tile per block 202 us; a thread per (tap, input
// channel) reading its input from global memory 972, 826 and 878 us.
template <int CI, int CO>
__global__ void __launch_bounds__(kWgradThreads, 1)
k_wgrad_tile(const float* __restrict__ X, const float* __restrict__ dY, int dil, TrainGrid g, bool vec,
             float* __restrict__ partial)
{
    constexpr int IG = CI / 4;           // lane groups of 4 input channels
    constexpr int CW = CO == 32 ? 8 : 2; // output channels per lane
    constexpr int CG = CO / CW;          // lane groups of output channels
    constexpr int PL = 32 / (IG * CG);   // pixels walked side by side
    constexpr int NW = 9 * CI * CO;
    extern __shared__ __align__(16) float sm[];
    const int hw = kTrainTile + 2 * dil;
    const int xsz = hw * hw * CI;
    constexpr int gsz = kTrainTile * kTrainTile * CO;
    float *xs = sm, *gs = sm + 2 * xsz; // two tiles [hw][hw][CI] of X, two [16][16][CO] of dY
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tr = warp % 3, rg = warp / 3;
    const int cg = lane % CG * CW, ig = lane / CG % IG * 4, pl = lane / (CG * IG);
    f2 acc[3][4][CW / 2];
    float bacc = 0.0f; // output channel threadIdx.x % CO (a divisor of the block's threads)
#pragma unroll
    for (int k = 0; k < CW / 2; ++k) {
#pragma unroll
        for (int i = 0; i < 12; ++i) acc[i / 4][i % 4][k] = f2_make(0.0f, 0.0f);
    }
    int64_t b, tile = blockIdx.x;
    int y0, x0, yn, xn;
    auto stage = [&](int64_t tl, int buf, int& ys, int& xo) {
        tile_origin(g, tl, b, ys, xo);
        if (tl < g.tiles) {
            stage_tile<CI, false>(X, g, b, ys, xo, dil, vec, xs + buf * xsz);
            stage_tile<CO, false>(dY, g, b, ys, xo, 0, true, gs + buf * gsz); // zeros outside the image
        }
        cp_async_commit();
    };
    stage(tile, 0, y0, x0);
    for (int cur = 0; tile < g.tiles; tile += gridDim.x, cur ^= 1) {
        stage(tile + gridDim.x, cur ^ 1, yn, xn);
        cp_async_wait<1>();
        __syncthreads();
#pragma unroll 8
        for (int i = threadIdx.x; i < gsz; i += kWgradThreads) bacc += gs[cur * gsz + i];
        const int rows = min(4, g.H - y0 - 4 * rg);
        const float* xr = xs + cur * xsz + ((4 * rg + dil + dil * (tr - 1)) * hw + pl) * CI + ig;
        const float* gr = gs + cur * gsz + (4 * rg * kTrainTile + pl) * CO + cg;
        auto pixel = [&](int x) {
            f2 d[CW / 2];
            if constexpr (CW == 8) {
                const ulonglong2 d0 = *reinterpret_cast<const ulonglong2*>(gr + x * CO);
                const ulonglong2 d1 = *reinterpret_cast<const ulonglong2*>(gr + x * CO + 4);
                d[0] = d0.x;
                d[1] = d0.y;
                d[2] = d1.x;
                d[3] = d1.y;
            }
            else {
                d[0] = *reinterpret_cast<const f2*>(gr + x * CO);
            }
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                const float4 q = *reinterpret_cast<const float4*>(xr + (x + dil * t) * CI);
                const float qa[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const f2 x2 = f2_make(qa[i], qa[i]);
#pragma unroll
                    for (int k = 0; k < CW / 2; ++k) acc[t][i][k] = f2_fma_acc(x2, d[k], acc[t][i][k]);
                }
            }
        };
        // pixels inside the image only: a zero of dY outside times an infinite or NaN neighbour would be NaN
        const int cols = g.W - x0;
        for (int y = 0; y < rows; ++y, xr += hw * CI, gr += kTrainTile * CO) {
            if (cols >= kTrainTile) {
#pragma unroll(PL == 1 ? 16 : 2)
                for (int x = 0; x < kTrainTile; x += PL) pixel(x);
            }
            else {
#pragma unroll 1
                for (int x = 0; x < cols - pl; x += PL) pixel(x);
            }
        }
        __syncthreads();
        y0 = yn;
        x0 = xn;
    }
    cp_async_wait<0>(); // (empty groups) before the buffers are reused
    // the pixel lanes' sums, fixed order
#pragma unroll
    for (int o = 16; o >= 32 / PL && PL > 1; o >>= 1) {
#pragma unroll
        for (int k = 0; k < CW / 2; ++k) {
#pragma unroll
            for (int i = 0; i < 12; ++i)
                acc[i / 4][i % 4][k] =
                    f2_add(acc[i / 4][i % 4][k], __shfl_xor_sync(0xffffffffu, acc[i / 4][i % 4][k], o));
        }
    }
    // the row groups' sums: [4][NW] in shared memory
    if (pl == 0) {
        float* o = sm + rg * NW;
#pragma unroll
        for (int t = 0; t < 3; ++t)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int k = 0; k < CW / 2; ++k)
                    *reinterpret_cast<f2*>(o + ((tr * 3 + t) * CI + ig + i) * CO + cg + 2 * k) = acc[t][i][k];
    }
    float* bs = sm + 4 * NW;
    bs[threadIdx.x] = bacc;
    __syncthreads();
    float* out = partial + static_cast<int64_t>(blockIdx.x) * (NW + CO);
    for (int i = threadIdx.x; i < NW; i += kWgradThreads)
        out[i] = ((sm[i] + sm[NW + i]) + sm[2 * NW + i]) + sm[3 * NW + i];
    if (threadIdx.x < CO) {
        float v = 0.0f;
        for (int i = threadIdx.x; i < kWgradThreads; i += CO) v += bs[i];
        out[NW + threadIdx.x] = v;
    }
}

// out[i] = sum over blocks of partial[b][i]: 8 runs of consecutive blocks, each summed in block
// order by one thread, then added in order (deterministic). 256 threads = 32 outputs x 8 runs.
__global__ void __launch_bounds__(256)
k_sum_partials(const float* __restrict__ partial, int nblk, int n, float* __restrict__ out)
{
    __shared__ float sh[8][33];
    const int l = threadIdx.x & 31, r = threadIdx.x >> 5;
    const int i = blockIdx.x * 32 + l;
    const int per = (nblk + 7) / 8, b0 = r * per, b1 = min(b0 + per, nblk);
    float s = 0.0f;
    if (i < n) {
#pragma unroll 8
        for (int b = b0; b < b1; ++b) s += partial[static_cast<int64_t>(b) * n + i];
    }
    sh[r][l] = s;
    __syncthreads();
    if (r == 0 && i < n) {
        float v = sh[0][l];
#pragma unroll
        for (int k = 1; k < 8; ++k) v += sh[k][l];
        out[i] = v;
    }
}

} // namespace nn
} // namespace gfgpu
