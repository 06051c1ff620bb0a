// Element-wise and reduction kernels of the learned warm start (U-Net), all
// NHWC with bf16 activations and fp32 weights/gradients.  The GEMM-shaped 3x3
// convolutions run on the tensor cores (arec_unet_conv.cu); everything here is
// memory-bound or small.
#include <cuda_bf16.h>
#include <stdint.h>

#include <algorithm>

#include "arec_internal.cuh"
#include "arec_unet.cuh"

namespace arecgb {
namespace unet {

__device__ __forceinline__ float bf(const __nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ __nv_bfloat16 tobf(float v) { return __float2bfloat16(v); }

static int blocks_for(size_t n) {
    size_t b = (n + 255) / 256;
    return (int)(b < 152 * 16 ? (b < 1 ? 1 : b) : 152 * 16);
}

#define GRID_STRIDE(i, n) \
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < (n); i += (size_t)gridDim.x * blockDim.x)

// ---- first layer: 1 -> 32 channels, 3x3, bias, ReLU (CUDA cores: 9 MACs per output) --------
// A warp takes 8 columns (lane / 4) x 32 channels (lane % 4: eight of them, their
// weights in registers) and runs down kInRows rows with a window of 3 x 3 inputs.
constexpr int kInC = 32, kInRows = 16;

struct InWindow {
    const float *col;  // the image's column wx, row 0
    int H, W, wx;
    float v[4][3];  // rows h - 1 .. h + 2 (the last one is on its way) from v[(h - h0) % 4] on

    // Row h of the window's columns (0 outside the image).
    __device__ __forceinline__ void row(float (&r)[3], int h) const {
        const float *p = col + (ptrdiff_t)h * W;
#pragma unroll
        for (int d = 0; d < 3; d++)
            r[d] = h >= 0 && h < H && wx + d > 0 && wx + d <= W ? __ldg(p + d - 1) : 0.f;
    }
    __device__ __forceinline__ bool inside(int h, int t) const {
        const int hh = h + t / 3 - 1, ww = wx + t % 3 - 1;
        return hh >= 0 && hh < H && ww >= 0 && ww < W;
    }
    __device__ __forceinline__ void start(int h0) {
#pragma unroll
        for (int i = 0; i < 3; i++) row(v[i], h0 - 1 + i);
    }
    // Tap t at the u-th row of four.
    __device__ __forceinline__ float tap(int u, int t) const { return v[(u + t / 3) & 3][t % 3]; }
};

// Strip `t` of an N x H x W stack: image, first column and row.
__device__ __forceinline__ void in_strip(size_t t, int H, int W, size_t &n, int &w0, int &h0) {
    const int wt = (W + 7) / 8, ht = (H + kInRows - 1) / kInRows;
    w0 = (int)(t % wt) * 8;
    h0 = (int)(t / wt % ht) * kInRows;
    n = t / wt / ht;
}
static size_t in_strips(int N, int H, int W) {
    return (size_t)N * ((W + 7) / 8) * ((H + kInRows - 1) / kInRows);
}

// Per output the FMAs run in tap order from the bias (taps outside the image
// skipped).  Bound by the issue of its instructions (288 multiply-adds per pixel, in
// pairs; the 64 bytes written per pixel would take 160 us at 16 x 1024^2): 438 us
// there; 752 with one thread per pixel and all channels, whose 288 weights came from
// shared memory for every pixel.  Rows take turns in the window's registers (a copy
// from one to the next would wait for the load in flight).
__global__ void __launch_bounds__(128, 4)
    k_conv_in(const float *__restrict__ x, const float *__restrict__ w, const float *__restrict__ b,
              __nv_bfloat16 *__restrict__ y, int N, int H, int W, size_t strips) {
    const int lane = threadIdx.x & 31, q = lane & 3;
    float2 sw[4][9], sb[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int c = q * 8 + 2 * j;
        sb[j] = make_float2(b[c], b[c + 1]);
#pragma unroll
        for (int t = 0; t < 9; t++) sw[j][t] = make_float2(w[c * 9 + t], w[(c + 1) * 9 + t]);
    }
    for (size_t s = (size_t)blockIdx.x * 4 + (threadIdx.x >> 5); s < strips; s += (size_t)gridDim.x * 4) {
        size_t n;
        int w0, h0;
        in_strip(s, H, W, n, w0, h0);
        InWindow win;
        win.H = H, win.W = W, win.wx = w0 + (lane >> 2);
        if (win.wx >= W) continue;
        const bool inner = w0 > 0 && w0 + 8 < W;  // all taps of the strip's columns
        win.col = x + n * H * W + win.wx;
        win.start(h0);
        for (int hu = h0; hu < min(H, h0 + kInRows); hu += 4)
#pragma unroll
          for (int u = 0; u < 4; u++) {
            const int h = hu + u;
            if (h >= H) break;
            win.row(win.v[(u + 3) & 3], h + 2);
            float2 o[4];
#pragma unroll
            for (int j = 0; j < 4; j++) o[j] = sb[j];
            const bool all = h > 0 && h + 1 < H && inner;  // uniform over the warp
            if (all) {
#pragma unroll
                for (int t = 0; t < 9; t++) {
                    const float2 v = make_float2(win.tap(u, t), win.tap(u, t));
#pragma unroll
                    for (int j = 0; j < 4; j++) o[j] = __ffma2_rn(sw[j][t], v, o[j]);
                }
            } else {
#pragma unroll
                for (int t = 0; t < 9; t++)
                    if (win.inside(h, t)) {
                        const float2 v = make_float2(win.tap(u, t), win.tap(u, t));
#pragma unroll
                        for (int j = 0; j < 4; j++) o[j] = __ffma2_rn(sw[j][t], v, o[j]);
                    }
            }
            __align__(16) __nv_bfloat162 r[4];
#pragma unroll
            for (int j = 0; j < 4; j++) r[j] = __floats2bfloat162_rn(fmaxf(o[j].x, 0.f), fmaxf(o[j].y, 0.f));
            *reinterpret_cast<uint4 *>(y + ((n * H + h) * W + win.wx) * kInC + q * 8) =
                *reinterpret_cast<const uint4 *>(r);
        }
    }
}

// Weight and bias gradient of the first layer from the gradient dy of its output y:
// with dpre = dy where y > 0, gw[c][t] += sum_p dpre[p][c] x[p + t], gb[c] += sum_p
// dpre[p][c] (pixels with dpre = 0 and taps outside the image skipped).  The sums of a
// thread's 8 channels stay in registers over its strips; the block adds them at the
// end, one FP32 atomic per value.  Bound by the reads of y and dy.  With a ReLU pass and a
// kernel with one channel per block 111 + 342 us at 16 x 256^2, now 96.
__global__ void __launch_bounds__(128, 4)
    k_conv_in_bwd(const float *__restrict__ x, const __nv_bfloat16 *__restrict__ y,
                  const __nv_bfloat16 *__restrict__ dy, float *__restrict__ gw, float *__restrict__ gb,
                  int N, int H, int W, size_t strips) {
    __shared__ float red[4][4][80];
    const int lane = threadIdx.x & 31, q = lane & 3, warp = threadIdx.x >> 5;
    float acc[8][10];
#pragma unroll
    for (int j = 0; j < 8; j++)
#pragma unroll
        for (int t = 0; t < 10; t++) acc[j][t] = 0.f;
    for (size_t s = (size_t)blockIdx.x * 4 + warp; s < strips; s += (size_t)gridDim.x * 4) {
        size_t n;
        int w0, h0;
        in_strip(s, H, W, n, w0, h0);
        InWindow win;
        win.H = H, win.W = W, win.wx = w0 + (lane >> 2);
        if (win.wx >= W) continue;
        win.col = x + n * H * W + win.wx;
        win.start(h0);
        for (int hu = h0; hu < min(H, h0 + kInRows); hu += 4)
#pragma unroll
          for (int u = 0; u < 4; u++) {
            const int h = hu + u;
            if (h >= H) break;
            win.row(win.v[(u + 3) & 3], h + 2);
            const size_t o = ((n * H + h) * W + win.wx) * kInC + q * 8;
            const uint4 yv = *reinterpret_cast<const uint4 *>(y + o);
            const uint4 dv = *reinterpret_cast<const uint4 *>(dy + o);
            const __nv_bfloat16 *yb = reinterpret_cast<const __nv_bfloat16 *>(&yv);
            const __nv_bfloat16 *db = reinterpret_cast<const __nv_bfloat16 *>(&dv);
            float d[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                d[j] = bf(yb[j]) > 0.f ? bf(db[j]) : 0.f;
                acc[j][9] += d[j];
            }
#pragma unroll
            for (int t = 0; t < 9; t++)
                if (win.inside(h, t)) {
#pragma unroll
                    for (int j = 0; j < 8; j++)
                        if (d[j] != 0.f) acc[j][t] = fmaf(d[j], win.tap(u, t), acc[j][t]);
                }
        }
    }
    // lanes of the same channels, then the block's warps
#pragma unroll
    for (int j = 0; j < 8; j++)
#pragma unroll
        for (int t = 0; t < 10; t++) {
            float v = acc[j][t];
            for (int o = 4; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane < 4) red[warp][q][j * 10 + t] = v;
        }
    __syncthreads();
    for (int i = threadIdx.x; i < 320; i += 128) {
        const int c = i / 10, t = i % 10;
        float v = 0.f;
        for (int k = 0; k < 4; k++) v += red[k][c / 8][c % 8 * 10 + t];
        atomicAdd(t < 9 ? &gw[c * 9 + t] : &gb[c], v);
    }
}

// ---- last layer: 1x1, C -> 1, plus the residual input --------------------------------------
template <int C>
__global__ void __launch_bounds__(256)
    k_conv_out(const __nv_bfloat16 *__restrict__ h, const float *__restrict__ w,
               const float *__restrict__ b, const float *__restrict__ x0,
               float *__restrict__ y, size_t P) {
    __shared__ float sw[C];
    for (int i = threadIdx.x; i < C; i += blockDim.x) sw[i] = w[i];
    __syncthreads();
    GRID_STRIDE(p, P) {
        float s = b[0] + x0[p];
        const uint4 *hp = reinterpret_cast<const uint4 *>(h + p * C);
#pragma unroll
        for (int q = 0; q < C / 8; q++) {
            const uint4 hv = hp[q];
            const __nv_bfloat16 *hb = reinterpret_cast<const __nv_bfloat16 *>(&hv);
#pragma unroll
            for (int j = 0; j < 8; j++) s = fmaf(sw[q * 8 + j], bf(hb[j]), s);
        }
        y[p] = s;
    }
}

// dh[p][c] = w[c]*dy[p]; gw[c] += sum dy*h; gb += sum dy  (C = kOutC channels)
constexpr int kOutC = 32;
__global__ void __launch_bounds__(128)
    k_conv_out_bwd(const __nv_bfloat16 *__restrict__ h, const float *__restrict__ w,
                   const float *__restrict__ dy, __nv_bfloat16 *__restrict__ dh,
                   float *__restrict__ gw, float *__restrict__ gb, size_t P) {
    __shared__ float sred[kOutC + 1][128];
    float acc[kOutC + 1];
#pragma unroll
    for (int c = 0; c <= kOutC; c++) acc[c] = 0.f;
    GRID_STRIDE(p, P) {
        const float d = dy[p];
        const uint4 *hp = reinterpret_cast<const uint4 *>(h + p * kOutC);
        uint4 *dp = reinterpret_cast<uint4 *>(dh + p * kOutC);
#pragma unroll
        for (int q = 0; q < kOutC / 8; q++) {
            const uint4 hv = hp[q];
            const __nv_bfloat16 *hb = reinterpret_cast<const __nv_bfloat16 *>(&hv);
            __align__(16) __nv_bfloat16 o[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                o[j] = tobf(w[q * 8 + j] * d);
                acc[q * 8 + j] = fmaf(d, bf(hb[j]), acc[q * 8 + j]);
            }
            dp[q] = *reinterpret_cast<const uint4 *>(o);
        }
        acc[kOutC] += d;
    }
#pragma unroll
    for (int c = 0; c <= kOutC; c++) sred[c][threadIdx.x] = acc[c];
    __syncthreads();
    for (int o = 64; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o)
            for (int c = 0; c <= kOutC; c++) sred[c][threadIdx.x] += sred[c][threadIdx.x + o];
        __syncthreads();
    }
    if ((int)threadIdx.x < kOutC) atomicAdd(&gw[threadIdx.x], sred[threadIdx.x][0]);
    if ((int)threadIdx.x == kOutC) atomicAdd(gb, sred[kOutC][0]);
}

// ---- pooling / upsampling / concat -----------------------------------------------------------
// 2x2 max pooling with the arg max (0..3, first of equals) per output; one
// thread per output pixel and 8 channels (16-byte vectors; C % 8 == 0).
__global__ void k_maxpool(const __nv_bfloat16 *__restrict__ x, __nv_bfloat16 *__restrict__ y,
                          uint8_t *__restrict__ arg, int N, int H, int W, int C, int xs) {
    const int Ho = H / 2, Wo = W / 2, C8 = C / 8;
    const size_t n_out = (size_t)N * Ho * Wo * C8;
    GRID_STRIDE(i, n_out) {
        const int g = (int)(i % C8);
        const size_t po = i / C8;
        const int wo = (int)(po % Wo);
        const size_t nho = po / Wo;  // n * Ho + ho
        const size_t top = (2 * nho) * W + 2 * wo;  // (n * H + 2 ho) * W + 2 wo
        float best[8];
        uint8_t bi[8];
#pragma unroll
        for (int t = 0; t < 4; t++) {
            const size_t pix = top + (size_t)(t >> 1) * W + (t & 1);
            const uint4 xv = *reinterpret_cast<const uint4 *>(x + pix * xs + g * 8);
            const __nv_bfloat16 *xb = reinterpret_cast<const __nv_bfloat16 *>(&xv);
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const float v = bf(xb[j]);
                if (t == 0 || v > best[j]) {
                    best[j] = v;
                    bi[j] = (uint8_t)t;
                }
            }
        }
        __align__(16) __nv_bfloat16 o[8];
#pragma unroll
        for (int j = 0; j < 8; j++) o[j] = tobf(best[j]);
        *reinterpret_cast<uint4 *>(y + po * C + g * 8) = *reinterpret_cast<const uint4 *>(o);
        if (arg) {
            uint2 a;
            a.x = bi[0] | (bi[1] << 8) | (bi[2] << 16) | ((uint32_t)bi[3] << 24);
            a.y = bi[4] | (bi[5] << 8) | (bi[6] << 16) | ((uint32_t)bi[7] << 24);
            *reinterpret_cast<uint2 *>(arg + po * C + g * 8) = a;
        }
    }
}

// Gradient of a level's skip tensor: dx = skip + (the pooled gradient dy at the arg
// max of its 2 x 2 pixels, 0 elsewhere), summed in FP32, one thread per pooled pixel
// and 8 channels.  Bound by its traffic (12 bytes per pooled value and pixel).  An
// FP32 accumulator cleared, added to twice and rounded took 90 + 56 + 60 us and a
// clearing pass at 16 x 256^2 x 32.
__global__ void k_skip_grad(const __nv_bfloat16 *__restrict__ skip, const __nv_bfloat16 *__restrict__ dy,
                            const uint8_t *__restrict__ arg, __nv_bfloat16 *__restrict__ dx, int N, int H,
                            int W, int C) {
    const int Ho = H / 2, Wo = W / 2, C8 = C / 8;
    const size_t n_out = (size_t)N * Ho * Wo * C8;
    GRID_STRIDE(i, n_out) {
        const int g = (int)(i % C8);
        const size_t po = i / C8;
        const int wo = (int)(po % Wo);
        const size_t top = (2 * (po / Wo)) * W + 2 * wo;
        const uint4 dv = *reinterpret_cast<const uint4 *>(dy + po * C + g * 8);
        const uint2 av = *reinterpret_cast<const uint2 *>(arg + po * C + g * 8);
        const __nv_bfloat16 *db = reinterpret_cast<const __nv_bfloat16 *>(&dv);
        const uint8_t *ab = reinterpret_cast<const uint8_t *>(&av);
#pragma unroll
        for (int t = 0; t < 4; t++) {
            const size_t o = (top + (size_t)(t >> 1) * W + (t & 1)) * C + g * 8;
            const uint4 sv = *reinterpret_cast<const uint4 *>(skip + o);
            const __nv_bfloat16 *sb = reinterpret_cast<const __nv_bfloat16 *>(&sv);
            __align__(16) __nv_bfloat16 r[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                float v = 0.f + bf(sb[j]);
                if (ab[j] == t) v += bf(db[j]);
                r[j] = tobf(v);
            }
            *reinterpret_cast<uint4 *>(dx + o) = *reinterpret_cast<const uint4 *>(r);
        }
    }
}

// nearest 2x upsampling of x [N][H][W][C] into channels [0, C) of y [N][2H][2W][Cy]
// One thread per input pixel and 8 channels: one 16-byte load, four stores
// (C, Cy multiples of 8).
__global__ void k_upsample(const __nv_bfloat16 *__restrict__ x, __nv_bfloat16 *__restrict__ y,
                           int N, int H, int W, int C, int Cy) {
    const int C8 = C / 8;
    const size_t n_in = (size_t)N * H * W * C8;
    GRID_STRIDE(i, n_in) {
        const int g = (int)(i % C8);
        const size_t p = i / C8;
        const int w = (int)(p % W);
        const size_t nh = p / W;  // n * H + h
        const uint4 v = *reinterpret_cast<const uint4 *>(x + p * C + g * 8);
        const size_t o0 = ((2 * nh) * (2 * W) + 2 * w) * Cy + g * 8;  // row 2h, column 2w
        *reinterpret_cast<uint4 *>(y + o0) = v;
        *reinterpret_cast<uint4 *>(y + o0 + Cy) = v;
        *reinterpret_cast<uint4 *>(y + o0 + (size_t)2 * W * Cy) = v;
        *reinterpret_cast<uint4 *>(y + o0 + (size_t)2 * W * Cy + Cy) = v;
    }
}

// dx[n][h][w][c] = sum over the 2x2 children of dy (channels [0, C) of a Cy-channel
// tensor); one thread per pixel and 8 channels (one channel each: 112 us at
// 16 x 128^2 x 64, a quarter of the sectors' bytes per load)
__global__ void k_upsample_bwd(const __nv_bfloat16 *__restrict__ dy, __nv_bfloat16 *__restrict__ dx,
                               int N, int H, int W, int C, int Cy) {
    const int C8 = C / 8;
    const size_t n_in = (size_t)N * H * W * C8;
    GRID_STRIDE(i, n_in) {
        const int g = (int)(i % C8);
        const size_t p = i / C8;
        const int w = (int)(p % W);
        const size_t nh = p / W;  // n * H + h
        const size_t o0 = ((2 * nh) * (2 * W) + 2 * w) * Cy + g * 8;  // row 2h, column 2w
        float s[8];
#pragma unroll
        for (int j = 0; j < 8; j++) s[j] = 0.f;
#pragma unroll
        for (int t = 0; t < 4; t++) {
            const uint4 v = *reinterpret_cast<const uint4 *>(dy + o0 + (size_t)(t >> 1) * 2 * W * Cy +
                                                             (t & 1) * Cy);
            const __nv_bfloat16 *b = reinterpret_cast<const __nv_bfloat16 *>(&v);
#pragma unroll
            for (int j = 0; j < 8; j++) s[j] += bf(b[j]);
        }
        __align__(16) __nv_bfloat16 r[8];
#pragma unroll
        for (int j = 0; j < 8; j++) r[j] = tobf(s[j]);
        *reinterpret_cast<uint4 *>(dx + p * C + g * 8) = *reinterpret_cast<const uint4 *>(r);
    }
}

// y [P][C] = channels [off, off + C) of x [P][Cx]
__global__ void k_chan_take(const __nv_bfloat16 *__restrict__ x, __nv_bfloat16 *__restrict__ y,
                            size_t P, int C, int Cx, int off) {
    const int C8 = C / 8;  // 16-byte vectors (C, Cx, off multiples of 8)
    GRID_STRIDE(i, P * C8) {
        const size_t p = i / C8;
        const int g = (int)(i % C8);
        *reinterpret_cast<uint4 *>(y + p * C + g * 8) =
            *reinterpret_cast<const uint4 *>(x + p * Cx + off + g * 8);
    }
}

__global__ void k_f32_to_bf16(const float *__restrict__ a, __nv_bfloat16 *__restrict__ b, size_t n) {
    GRID_STRIDE(i, n) { b[i] = tobf(a[i]); }
}

// dpre = dy * (y > 0) (ReLU backward on the post-activation output; row strides) and
// the bias gradient gb[c] += sum_p dpre[p][c].
// One thread per pixel and 8 channels (16-byte vectors); a thread keeps its
// channels over its pixels, so the sums stay in registers until the block adds
// them (FP32, one atomic per channel and block).  C a power of two in [32, 256].
__global__ void __launch_bounds__(256)
    k_relu_bwd_bias(const __nv_bfloat16 *__restrict__ y, int yys,
                    const __nv_bfloat16 *__restrict__ dy, int dys,
                    __nv_bfloat16 *__restrict__ dpre, float *__restrict__ gb, size_t P, int C) {
    __shared__ float red[256][9];
    const int C8 = C / 8, g = threadIdx.x & (C8 - 1), per = 256 / C8;
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; j++) acc[j] = 0.f;
    for (size_t p = (size_t)blockIdx.x * per + threadIdx.x / C8; p < P;
         p += (size_t)gridDim.x * per) {
        const uint4 yv = *reinterpret_cast<const uint4 *>(y + p * yys + g * 8);
        const uint4 dv = *reinterpret_cast<const uint4 *>(dy + p * dys + g * 8);
        const __nv_bfloat16 *yb = reinterpret_cast<const __nv_bfloat16 *>(&yv);
        const __nv_bfloat16 *db = reinterpret_cast<const __nv_bfloat16 *>(&dv);
        __align__(16) __nv_bfloat16 o[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            o[j] = bf(yb[j]) > 0.f ? db[j] : tobf(0.f);
            acc[j] += bf(o[j]);
        }
        *reinterpret_cast<uint4 *>(dpre + p * C + g * 8) = *reinterpret_cast<const uint4 *>(o);
    }
#pragma unroll
    for (int j = 0; j < 8; j++) red[threadIdx.x][j] = acc[j];
    __syncthreads();
    if ((int)threadIdx.x < C) {
        const int gg = threadIdx.x / 8, j = threadIdx.x % 8;
        float s = 0.f;
        for (int t = gg; t < 256; t += C8) s += red[t][j];
        atomicAdd(&gb[threadIdx.x], s);
    }
}

// Data-gradient weights: wt[ci][t][co] = w[co][8 - t][ci] (flip and transpose), bf16.
__global__ void k_flip_weights(const float *__restrict__ w, __nv_bfloat16 *__restrict__ wt, int Cin,
                               int Cout) {
    GRID_STRIDE(i, (size_t)Cout * 9 * Cin) {
        const int ci = (int)(i % Cin);
        const int t = (int)((i / Cin) % 9);
        const int co = (int)(i / ((size_t)Cin * 9));
        wt[((size_t)ci * 9 + (8 - t)) * Cout + co] = tobf(w[i]);
    }
}

// Loss: mean squared error over n values; writes d(loss)/d(out) and the sum of
// squared errors (one partial per block).
__global__ void k_mse(const float *__restrict__ out, const float *__restrict__ target,
                      float *__restrict__ dout, double *__restrict__ partial, size_t n, float scale) {
    __shared__ double red[256];
    double s = 0.0;
    GRID_STRIDE(i, n) {
        const float d = out[i] - target[i];
        dout[i] = scale * 2.f * d;
        s += (double)d * d;
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = red[0];
}

// Multi-scale loss: level s of the error pyramid is the error out - target
// averaged over 2^s x 2^s blocks (level 0 the error itself).  Pooling by 2 of
// level s-1 into level s; level 1 is pooled straight from out - target.
__global__ void k_err_pool(const float *__restrict__ a, const float *__restrict__ b,
                           float *__restrict__ y, int N, int H, int W) {
    const int Ho = H / 2, Wo = W / 2;
    GRID_STRIDE(p, (size_t)N * Ho * Wo) {
        const int xo = (int)(p % Wo), yo = (int)((p / Wo) % Ho), n = (int)(p / ((size_t)Wo * Ho));
        const size_t i0 = ((size_t)n * H + 2 * yo) * W + 2 * xo;
        float s = a[i0] + a[i0 + 1] + a[i0 + W] + a[i0 + W + 1];
        if (b) s -= b[i0] + b[i0 + 1] + b[i0 + W] + b[i0 + W + 1];
        y[p] = 0.25f * s;
    }
}

// dout = scale * 2 * sum_s alpha_s * level_s(block of p), alpha_s = ratio^s;
// the loss sum_s alpha_s * mean(level_s^2) is accumulated per pixel as
// sum_s alpha_s * level_s(block of p)^2 (the caller divides by the pixels).
__global__ void k_multiscale_grad(const float *__restrict__ out, const float *__restrict__ target,
                                  const float *__restrict__ pyr, float *__restrict__ dout,
                                  double *__restrict__ partial, int N, int H, int W, int levels,
                                  float ratio, float scale) {
    __shared__ double red[256];
    double acc = 0.0;
    GRID_STRIDE(p, (size_t)N * H * W) {
        const int x = (int)(p % W), yy = (int)((p / W) % H), n = (int)(p / ((size_t)W * H));
        const float e = out[p] - target[p];
        float g = e, a = 1.0f;
        double l = (double)e * e;
        const float *lev = pyr;
        int h = H, w = W;
        for (int s = 1; s <= levels; s++) {
            h >>= 1;
            w >>= 1;
            a *= ratio;
            const float v = lev[((size_t)n * h + (yy >> s)) * w + (x >> s)];
            g += a * v;
            // summed over the cell's 4^s pixels and divided by P: the cell mean
            l += (double)a * v * v;
            lev += (size_t)N * h * w;
        }
        dout[p] = scale * 2.f * g;
        acc += l;
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = red[0];
}

// AdamW on fp32 master weights; refreshes the bf16 copy.
__global__ void k_adamw(float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m,
                        float *__restrict__ v, size_t n, float lr, float b1, float b2, float eps,
                        float wd, float bc1, float bc2) {
    GRID_STRIDE(i, n) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float mh = mi / bc1, vh = vi / bc2;
        w[i] = w[i] - lr * (mh / (sqrtf(vh) + eps) + wd * w[i]);
    }
}

// Cylinder volume [nrays][ys] (slices y0..y0+B) <-> image stack [B][np][np]
// (iz rows, ix columns, np >= nx padded with zeros), scaled by `scale`; zeros
// outside the disk (the device form of ImageCyl2CB / ImageCB2Cyl,
// AREC3D/AREC3D/arecImage.cpp:88-232).
__global__ void k_cyl_to_img(const float *__restrict__ vol, const RowInfo *__restrict__ rows,
                             float *__restrict__ img, int nx, int npad, int ys, int y0, int B,
                             float scale) {
    GRID_STRIDE(i, (size_t)B * npad * npad) {
        const int ix = (int)(i % npad), iz = (int)((i / npad) % npad);
        const int b = (int)(i / ((size_t)npad * npad));
        float v = 0.f;
        if (iz < nx) {
            const RowInfo r = rows[iz];
            if (ix >= r.lo && ix <= r.hi)
                v = scale * vol[(size_t)(r.start + ix - r.lo) * ys + y0 + b];
        }
        img[i] = v;
    }
}

__global__ void k_img_to_cyl(const float *__restrict__ img, const RowInfo *__restrict__ rows,
                             float *__restrict__ vol, int nx, int npad, int ys, int y0, int B,
                             float scale) {
    GRID_STRIDE(i, (size_t)B * npad * npad) {
        const int ix = (int)(i % npad), iz = (int)((i / npad) % npad);
        const int b = (int)(i / ((size_t)npad * npad));
        if (iz < nx) {
            const RowInfo r = rows[iz];
            if (ix >= r.lo && ix <= r.hi)
                vol[(size_t)(r.start + ix - r.lo) * ys + y0 + b] = scale * img[i];
        }
    }
}

// Sum of squares of n floats, one FP64 partial per block (summed on the host).
__global__ void k_sumsq_partial(const float *__restrict__ a, size_t n, double *__restrict__ part) {
    __shared__ double red[256];
    double s = 0.0;
    GRID_STRIDE(i, n) s += (double)a[i] * a[i];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

// ---- host launchers -----------------------------------------------------------------------
void conv_in(const float *x, const float *w, const float *b, __nv_bfloat16 *y, int N, int H, int W,
             int C, cudaStream_t st) {
    if (C != kInC) return;  // the network's first layer (32 channels)
    const size_t strips = in_strips(N, H, W);
    k_conv_in<<<(int)std::min<size_t>((strips + 3) / 4, 152 * 16), 128, 0, st>>>(x, w, b, y, N, H, W, strips);
}
void conv_in_bwd(const float *x, const __nv_bfloat16 *y, const __nv_bfloat16 *dy, float *gw, float *gb,
                 int N, int H, int W, int C, cudaStream_t st) {
    if (C != kInC) return;
    const size_t strips = in_strips(N, H, W);
    k_conv_in_bwd<<<(int)std::min<size_t>((strips + 3) / 4, 152 * 4), 128, 0, st>>>(x, y, dy, gw, gb, N, H,
                                                                                    W, strips);
}
void conv_out(const __nv_bfloat16 *h, const float *w, const float *b, const float *x0, float *y,
              size_t P, int C, cudaStream_t st) {
    if (C != kOutC) return;
    k_conv_out<kOutC><<<blocks_for(P), 256, 0, st>>>(h, w, b, x0, y, P);
}
void conv_out_bwd(const __nv_bfloat16 *h, const float *w, const float *dy, __nv_bfloat16 *dh,
                  float *gw, float *gb, size_t P, int C, cudaStream_t st) {
    (void)C;  // kOutC
    int blocks = (int)std::min<size_t>(1024, (P + 127) / 128);
    k_conv_out_bwd<<<blocks, 128, 0, st>>>(h, w, dy, dh, gw, gb, P);
}
// x: [N][H][W] pixels of xs channels (xs = 0: C), the first C of them pooled
void maxpool(const __nv_bfloat16 *x, __nv_bfloat16 *y, uint8_t *arg, int N, int H, int W, int C,
             cudaStream_t st, int xs) {
    k_maxpool<<<blocks_for((size_t)N * H * W * C / 32), 256, 0, st>>>(x, y, arg, N, H, W, C,
                                                                      xs > 0 ? xs : C);
}
void skip_grad(const __nv_bfloat16 *skip, const __nv_bfloat16 *dy, const uint8_t *arg, __nv_bfloat16 *dx,
               int N, int H, int W, int C, cudaStream_t st) {
    k_skip_grad<<<blocks_for((size_t)N * H * W * C / 32), 256, 0, st>>>(skip, dy, arg, dx, N, H, W, C);
}
void upsample(const __nv_bfloat16 *x, __nv_bfloat16 *y, int N, int H, int W, int C, int Cy,
              cudaStream_t st) {
    k_upsample<<<blocks_for((size_t)N * H * W * C / 8), 256, 0, st>>>(x, y, N, H, W, C, Cy);
}
void upsample_bwd(const __nv_bfloat16 *dy, __nv_bfloat16 *dx, int N, int H, int W, int C, int Cy,
                  cudaStream_t st) {
    k_upsample_bwd<<<blocks_for((size_t)N * H * W * C / 8), 256, 0, st>>>(dy, dx, N, H, W, C, Cy);
}
void chan_take(const __nv_bfloat16 *x, __nv_bfloat16 *y, size_t P, int C, int Cx, int off,
               cudaStream_t st) {
    k_chan_take<<<blocks_for(P * C / 8), 256, 0, st>>>(x, y, P, C, Cx, off);
}
void f32_to_bf16(const float *a, __nv_bfloat16 *b, size_t n, cudaStream_t st) {
    k_f32_to_bf16<<<blocks_for(n), 256, 0, st>>>(a, b, n);
}
void relu_bwd_bias(const __nv_bfloat16 *y, int yys, const __nv_bfloat16 *dy, int dys,
                   __nv_bfloat16 *dpre, float *gb, size_t P, int C, cudaStream_t st) {
    // about 16 pixels per thread at least, 8 blocks per SM at most
    const size_t per = 256 / (C / 8);
    const int blocks = (int)std::max<size_t>(1, std::min<size_t>(152 * 8, P / (16 * per)));
    k_relu_bwd_bias<<<blocks, 256, 0, st>>>(y, yys, dy, dys, dpre, gb, P, C);
}
void flip_weights(const float *w, __nv_bfloat16 *wt, int Cin, int Cout, cudaStream_t st) {
    k_flip_weights<<<blocks_for((size_t)Cout * 9 * Cin), 256, 0, st>>>(w, wt, Cin, Cout);
}
void mse(const float *out, const float *target, float *dout, double *partial, size_t n, float scale,
         int nblocks, cudaStream_t st) {
    k_mse<<<nblocks, 256, 0, st>>>(out, target, dout, partial, n, scale);
}
void multiscale_loss(const float *out, const float *target, float *pyr, float *dout,
                     double *partial, int N, int H, int W, int levels, float ratio, float scale,
                     int nblocks, cudaStream_t st) {
    float *lev = pyr;
    const float *prev = nullptr;
    int h = H, w = W;
    for (int s = 1; s <= levels; s++) {
        const size_t n = (size_t)N * (h / 2) * (w / 2);
        if (s == 1)
            k_err_pool<<<blocks_for(n), 256, 0, st>>>(out, target, lev, N, h, w);
        else
            k_err_pool<<<blocks_for(n), 256, 0, st>>>(prev, nullptr, lev, N, h, w);
        prev = lev;
        lev += n;
        h /= 2;
        w /= 2;
    }
    k_multiscale_grad<<<nblocks, 256, 0, st>>>(out, target, pyr, dout, partial, N, H, W, levels,
                                               ratio, scale);
}
void adamw(float *w, const float *g, float *m, float *v, size_t n, float lr, float b1, float b2,
           float eps, float wd, float bc1, float bc2, cudaStream_t st) {
    k_adamw<<<blocks_for(n), 256, 0, st>>>(w, g, m, v, n, lr, b1, b2, eps, wd, bc1, bc2);
}
void cyl_to_img(const float *vol, const RowInfo *rows, float *img, int nx, int npad, int ys,
                int y0, int B, float scale, cudaStream_t st) {
    k_cyl_to_img<<<blocks_for((size_t)B * npad * npad), 256, 0, st>>>(vol, rows, img, nx, npad, ys,
                                                                      y0, B, scale);
}
void img_to_cyl(const float *img, const RowInfo *rows, float *vol, int nx, int npad, int ys,
                int y0, int B, float scale, cudaStream_t st) {
    k_img_to_cyl<<<blocks_for((size_t)B * npad * npad), 256, 0, st>>>(img, rows, vol, nx, npad, ys,
                                                                      y0, B, scale);
}
void sumsq_partial(const float *a, size_t n, double *part, int nblocks, cudaStream_t st) {
    k_sumsq_partial<<<nblocks, 256, 0, st>>>(a, n, part);
}

}  // namespace unet
}  // namespace arecgb
