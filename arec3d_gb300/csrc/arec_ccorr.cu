// FFT cross-correlation shift search (reference arecCCImages,
// AREC3D/AREC3D/arecImage.cpp:384-434 = ccorr2d + speak per image pair,
// AREC3D/AREC3D/align2dstack.cpp:480-521, 1059-1166) and the Fourier shift
// (fshift2d, align2dstack.cpp:566-630).
//
//   c = IDFT2( conj(DFT2 x) * DFT2 y )   (unnormalised, [ny][nx], real)
//   peak = speak(c): |c| argmax with the reference's scan-order rules,
//          3x3 paraboloid fit, wrap to (-n/2, n/2].
//
// Pipeline per batch of image pairs (all FP32, sizes 2..4096 whose prime
// factors are 2, 3, 5 and 7), H = nx/2+1:
//   1. rows:    z = x + i*y, complex FFT of each row (one transform gives the
//               row spectra of both real images), split into the half spectra
//               S[ny][H] = (X, Y), interleaved.
//   2. columns: column FFTs of X and Y in step, C = conj(X)*Y, inverse column
//               FFT -> W[ny][H].
//   3. rows:    two Hermitian rows a, b as one complex inverse FFT of
//               A + i*B: c rows a (real part) and b (imaginary part), with
//               per-row peak statistics fused.
//   4. peak:    one block per pair reduces the row statistics exactly in the
//               reference's x-major scan order and fits the paraboloid in FP64.
// The Fourier shift runs the same row passes on pairs of rows of one image and
// a column pass that multiplies the phase factor.
//
// The transforms (arec_fft.cuh) keep 16 points per thread in registers: a pass
// reads its lines once and writes them once, so what is left is the traffic of
// the three passes (36 bytes per pixel of a pair: 8 + 8 rows, 8 + 4 columns,
// 4 + 4 rows; the Fourier shift 24).  Against Stockham passes that staged every
// line in shared memory first and last, gathered 16 scattered twiddles per
// butterfly and spilled (one block per SM), whole calls: 48 pairs of 2048^2
// 9.36 -> 2.52 ms, 30 pairs of 750 x 1000 1.89 -> 0.89 ms, the shift of 180
// images of 512^2 (then full complex spectra) 4.89 -> 0.53 ms; with the
// scratch from a pool 2.24, 0.59 and 0.31 ms.
#include <math.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <map>
#include <mutex>
#include <vector>

#include "arec_fft.cuh"
#include "arec_internal.cuh"

namespace arecgb {

using fft::FastDiv;
using fft::fdiv;
using fft::Passes;
using fft::plen;
using fft::Pow2;
using fft::pz;

// Lengths whose prime factors are 2, 3, 5 and 7 (the reference's FFTW takes any
// length; these cover the detector and crop sizes the alignment sees).
static inline bool smooth_length(int n) {
    if (n < 2 || n > 4096) return false;
    const int primes[4] = {2, 3, 5, 7};
    for (int p : primes)
        while (n % p == 0) n /= p;
    return n == 1;
}

// Lines of length n per block of the row passes (16 points per thread).
__device__ __host__ __forceinline__ int lines_per_block(int n) {
    return n >= fft::kElems ? 1 : fft::kElems / n;
}
static inline bool pow2_length(int n) { return n >= 16 && (n & (n - 1)) == 0; }
// Columns per block of a column pass over points of `w` bytes: the largest
// power of two with 4096 points per block; the run-time lengths hold two
// buffers and take 4096 points of 8 bytes or 2048 of 16 (about 70 KB, three
// blocks per SM).
static inline int col_tile(int ny, int w) {
    const int cap = pow2_length(ny) || w == 8 ? fft::kElems : fft::kElems / 2;
    int ct = 1;
    while (2 * ct * ny <= cap) ct *= 2;
    return ct;
}
// Stride between a column tile's lines in shared memory, in points of `w`
// bytes (u of them in 128 bytes): a warp reads ct lines x 32/ct consecutive
// points, so the lines start u / ct points apart modulo u; tiles of u lines or
// more take any odd stride.
__device__ __host__ __forceinline__ constexpr int col_stride(int n, int ct, int w) {
    const int u = 128 / w;
    return ct < u ? (plen(n) + u - 1) / u * u + u / ct : (plen(n) | 1);
}

// What a row pass transforms: pairs of images (shift search) or pairs of rows
// of one image (Fourier shift).
enum RowMode { kPairs = 0, kRows = 1 };

// ---------------------------------------------------------------------------
// Row passes, forward.  kPairs: z = x + i y per row, S[row][k] = (X, Y) as one
// float4.  kRows: z = row 2l + i row 2l+1, F[row][k] as float2.
// N > 0: a power of two; N = 0: `P`'s run-time length.
struct RowSpectra {
    float4 *S;   // kPairs: [nz][ny][H]
    float2 *F;   // kRows:  [nz][ny][H]
};

template <int MODE>
__device__ __forceinline__ void store_split(const RowSpectra &o, size_t img_row, int row, int ny,
                                            int H, int k, float2 Z, float2 Zm) {
    const float2 X = make_float2(0.5f * (Z.x + Zm.x), 0.5f * (Z.y - Zm.y));
    const float2 Y = make_float2(0.5f * (Z.y + Zm.y), -0.5f * (Z.x - Zm.x));
    if constexpr (MODE == kPairs) {
        o.S[img_row * H + k] = make_float4(X.x, X.y, Y.x, Y.y);
    } else {
        o.F[img_row * H + k] = X;
        if (row + 1 < ny) o.F[(img_row + 1) * H + k] = Y;
    }
}

template <int N, int MODE>
__global__ void __launch_bounds__(fft::kThreads, 3)
    k_rows_fwd(const float *__restrict__ x, const float *__restrict__ y, RowSpectra o, int nx,
               int ny, Passes P, FastDiv dH, const float2 *__restrict__ tw) {
    extern __shared__ float4 sm4[];
    float2 *sm = reinterpret_cast<float2 *>(sm4);
    const int n = N > 0 ? N : nx, H = n / 2 + 1;
    const int G = N > 0 ? Pow2<N ? N : 16>::G : lines_per_block(n);
    const int line0 = blockIdx.x * G, LS = plen(n);
    const size_t img = (size_t)blockIdx.y * ny;  // first row of the image
    const float *xi = x + img * n, *yi = MODE == kPairs ? y + img * n : x + img * n;
    auto load = [&](int line, int i) -> float2 {
        const int l = line0 + line;
        if constexpr (MODE == kPairs)
            return l < ny ? make_float2(xi[(size_t)l * n + i], yi[(size_t)l * n + i])
                          : make_float2(0.f, 0.f);
        else
            return make_float2(2 * l < ny ? xi[(size_t)(2 * l) * n + i] : 0.f,
                               2 * l + 1 < ny ? xi[(size_t)(2 * l + 1) * n + i] : 0.f);
    };
    if constexpr (N > 0) {
        using L2 = Pow2<N>;
        constexpr int TPL = L2::TPL, Ra = L2::template radix<false>(0);
        constexpr int Rl = L2::template radix<false>(L2::P - 1);
        constexpr bool WARP = TPL <= 32;
        const int line = threadIdx.x / TPL, b = threadIdx.x % TPL;
        float2 *L = sm + (size_t)line * LS;
        float2 v[1][16];
#pragma unroll
        for (int i = 0; i < 16 / Ra; i++)
#pragma unroll
            for (int r = 0; r < Ra; r++) v[0][i * Ra + r] = load(line, b + i * TPL + r * (N / Ra));
        fft::transform<N, false, WARP, 1>(v, L, b, tw);
        fft::exchange_sync<WARP>();
#pragma unroll
        for (int i = 0; i < 16 / Rl; i++)
#pragma unroll
            for (int r = 0; r < Rl; r++) L[pz(b + i * TPL + r * (N / Rl))] = v[0][i * Rl + r];
        fft::exchange_sync<WARP>();
        const int row = MODE == kPairs ? line0 + line : 2 * (line0 + line);
        if (row >= ny) return;
#pragma unroll
        for (int i = 0; i < 16 / Rl; i++)
#pragma unroll
            for (int r = 0; r <= Rl / 2; r++) {
                const int j = b + i * TPL, k = j + r * (N / Rl);
                if (r < Rl / 2 || j == 0)
                    store_split<MODE>(o, img + row, row, ny, H, k, v[0][i * Rl + r],
                                      L[pz((N - k) & (N - 1))]);
            }
    } else {
        fft::mixed_fill<false>(n, P.dn, G, 0, sm, LS, load);
        const float2 *z = fft::mixed_transform<1, false>(P, G, 0, sm, sm + G * LS, LS, tw);
        for (int t = threadIdx.x; t < G * H; t += fft::kThreads) {
            const int line = fdiv(t, dH), k = t - line * H;
            const int row = MODE == kPairs ? line0 + line : 2 * (line0 + line);
            if (row < ny)
                store_split<MODE>(o, img + row, row, ny, H, k, z[line * LS + pz(k)],
                                  z[line * LS + pz(k ? n - k : 0)]);
        }
    }
}

// ---------------------------------------------------------------------------
// Column pass of the shift search: ct columns of S per block; W = IDFT_col(
// conj(X)*Y).  The inverse transform starts on the registers the forward ones
// end with (its radices in reversed order).
__device__ __forceinline__ float2 conj_product(float2 a, float2 b) {
    // conj(conj(a) * b): the inverse transform is conj DFT conj
    return make_float2(a.x * b.x + a.y * b.y, -(a.x * b.y - a.y * b.x));
}

template <int N>
__global__ void __launch_bounds__(fft::kThreads, 2)
    k_cc_cols(const float4 *__restrict__ S, float2 *__restrict__ W, int nx, int ny, int ct, int lg,
              Passes P, const float2 *__restrict__ tw, const float2 *__restrict__ twr) {
    extern __shared__ float4 sm4[];
    float2 *sm2 = reinterpret_cast<float2 *>(sm4);
    const int n = N > 0 ? N : ny, H = nx / 2 + 1;
    const int c0 = blockIdx.x * ct;
    const size_t img = (size_t)blockIdx.y * n;
    const int LS4 = col_stride(n, ct, 16), LS2 = col_stride(n, ct, 8);
    auto load = [&](int c, int row) -> float4 {
        return c0 + c < H ? S[(img + row) * H + c0 + c] : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    if constexpr (N > 0) {
        using L2 = Pow2<N>;
        constexpr int TPL = L2::TPL, CT = L2::G, Ra = L2::template radix<false>(0);
        const int c = threadIdx.x % CT, b = threadIdx.x / CT;
        float2 v[2][16];
#pragma unroll
        for (int i = 0; i < 16 / Ra; i++)
#pragma unroll
            for (int r = 0; r < Ra; r++) {
                const float4 q = load(c, b + i * TPL + r * (N / Ra));
                v[0][i * Ra + r] = make_float2(q.x, q.y);
                v[1][i * Ra + r] = make_float2(q.z, q.w);
            }
        fft::transform<N, false, false, 2>(v, sm4 + c * LS4, b, tw);
        float2 w[1][16];
#pragma unroll
        for (int i = 0; i < 16; i++) w[0][i] = conj_product(v[0][i], v[1][i]);
        __syncthreads();  // the lines' layout changes
        fft::transform<N, true, false, 1>(w, sm2 + c * LS2, b, twr);
        if (c0 + c >= H) return;
#pragma unroll
        for (int i = 0; i < 16 / Ra; i++)
#pragma unroll
            for (int r = 0; r < Ra; r++) {
                const float2 z = w[0][i * Ra + r];
                W[(img + b + i * TPL + r * (N / Ra)) * H + c0 + c] = make_float2(z.x, -z.y);
            }
    } else {
        fft::mixed_fill<true>(n, P.dn, ct, lg, sm4, LS4, load);
        float4 *z4 = fft::mixed_transform<2, true>(P, ct, lg, sm4, sm4 + ct * LS4, LS4, tw);
        // the products stay in the slots of X (the inverse transform strides
        // over float4 slots)
        for (int t = threadIdx.x; t < ct * n; t += fft::kThreads) {
            float4 &q = z4[(t & (ct - 1)) * LS4 + pz(t >> lg)];
            const float2 z = conj_product(make_float2(q.x, q.y), make_float2(q.z, q.w));
            q.x = z.x;
            q.y = z.y;
        }
        __syncthreads();
        z4 = fft::mixed_transform<1, true>(P, ct, lg, z4, z4 == sm4 ? sm4 + ct * LS4 : sm4, LS4, tw);
        fft::mixed_drain<true>(n, P.dn, ct, lg, z4, LS4, [&](int c, int i, float4 z) {
            if (c0 + c < H) W[(img + i) * H + c0 + c] = make_float2(z.x, -z.y);
        });
    }
}

struct RowStat {
    float m;   // max |c| over the row
    int xpos;  // first x with c == +m (INT_MAX if none)
    int xneg;  // last x with c == -m (-1 if none)
    int pad;
};

// Combine two row statistics in favour of the reference's scan order.
__device__ __forceinline__ RowStat stat_merge(RowStat a, RowStat b) {
    if (b.m > a.m) return b;
    if (a.m > b.m) return a;
    RowStat r = a;
    r.xpos = min(a.xpos, b.xpos);
    r.xneg = max(a.xneg, b.xneg);
    return r;
}

// The statistics of one value at x (NaN never wins).
__device__ __forceinline__ RowStat stat_of(float v, int x) {
    const float a = fabsf(v);
    if (!(a == a)) return RowStat{-1.0f, INT_MAX, -1, 0};
    return RowStat{a, v == a ? x : INT_MAX, v == -a && v != a ? x : -1, 0};
}

__device__ __forceinline__ RowStat stat_warp(RowStat s) {
    for (int o = 16; o > 0; o >>= 1) {
        RowStat t;
        t.m = __shfl_down_sync(0xffffffffu, s.m, o);
        t.xpos = __shfl_down_sync(0xffffffffu, s.xpos, o);
        t.xneg = __shfl_down_sync(0xffffffffu, s.xneg, o);
        t.pad = 0;
        s = stat_merge(s, t);
    }
    return s;
}

// ---------------------------------------------------------------------------
// Row passes, inverse: rows a = 2l and b = 2l+1 of the half spectra W as one
// complex transform of A + i B (A, B real: their spectra Hermitian, so the
// zero and Nyquist terms are real).  kPairs: c rows and their peak
// statistics; kRows: out rows divided by nx*ny.
template <int N, int MODE>
__global__ void __launch_bounds__(fft::kThreads, 3)
    k_rows_inv(const float2 *__restrict__ W, float *__restrict__ c, RowStat *__restrict__ stats,
               int nx, int ny, Passes P, const float2 *__restrict__ tw) {
    extern __shared__ float4 sm4[];
    float2 *sm = reinterpret_cast<float2 *>(sm4);
    __shared__ unsigned s_m[512];
    __shared__ int s_pos[512], s_neg[512];
    const int n = N > 0 ? N : nx, H = n / 2 + 1;
    const int G = N > 0 ? Pow2<N ? N : 16>::G : lines_per_block(n);
    const int line0 = blockIdx.x * G, LS = plen(n);
    const size_t img = (size_t)blockIdx.y * ny;
    const float scale = (float)(nx * ny);
    auto load = [&](int line, int i) -> float2 {
        const int row = 2 * (line0 + line);
        const bool up = 2 * i > n;  // conj(Z[n - i]) of the Hermitian rows
        const int k = up ? n - i : i;
        const float2 *w = W + (img + row) * H + k;
        float2 a = row < ny ? w[0] : make_float2(0.f, 0.f);
        float2 b = row + 1 < ny ? w[H] : make_float2(0.f, 0.f);
        if (i == 0 || 2 * i == n) a.y = b.y = 0.f;
        // conj(A + i B): the inverse transform is conj DFT conj
        return up ? make_float2(a.x + b.y, a.y - b.x) : make_float2(a.x - b.y, -(a.y + b.x));
    };
    if constexpr (N > 0) {
        using L2 = Pow2<N>;
        constexpr int TPL = L2::TPL, Ra = L2::template radix<false>(0);
        constexpr int Rl = L2::template radix<false>(L2::P - 1);
        const int line = threadIdx.x / TPL, b = threadIdx.x % TPL;
        float2 v[1][16];
#pragma unroll
        for (int i = 0; i < 16 / Ra; i++)
#pragma unroll
            for (int r = 0; r < Ra; r++) v[0][i * Ra + r] = load(line, b + i * TPL + r * (N / Ra));
        fft::transform<N, false, (TPL <= 32), 1>(v, sm + (size_t)line * LS, b, tw);
        const int row = 2 * (line0 + line);
        const bool ra = row < ny, rb = row + 1 < ny;
        float *ca = c + (img + row) * n;
        if constexpr (MODE == kRows) {
#pragma unroll
            for (int i = 0; i < 16 / Rl; i++)
#pragma unroll
                for (int r = 0; r < Rl; r++) {
                    const int x = b + i * TPL + r * (N / Rl);
                    const float2 z = v[0][i * Rl + r];
                    if (ra) ca[x] = z.x / scale;
                    if (rb) ca[n + x] = -z.y / scale;
                }
        } else {
            // per row: max |c| (as an ordered integer; NaN never wins), then
            // the first x of +max and the last of -max
            for (int t = threadIdx.x; t < 2 * G; t += fft::kThreads) {
                s_m[t] = 0u;
                s_pos[t] = INT_MAX;
                s_neg[t] = -1;
            }
            unsigned ma = 0u, mb = 0u;
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const unsigned ua = __float_as_uint(fabsf(v[0][i].x));
                const unsigned ub = __float_as_uint(fabsf(v[0][i].y));
                ma = max(ma, ua > 0x7f800000u ? 0u : ua);
                mb = max(mb, ub > 0x7f800000u ? 0u : ub);
            }
            if constexpr (TPL >= 32) {
                ma = __reduce_max_sync(0xffffffffu, ma);
                mb = __reduce_max_sync(0xffffffffu, mb);
            }
            __syncthreads();
            if (TPL < 32 || (threadIdx.x & 31) == 0) {
                atomicMax(&s_m[2 * line], ma);
                atomicMax(&s_m[2 * line + 1], mb);
            }
            __syncthreads();
            const unsigned Ma = s_m[2 * line], Mb = s_m[2 * line + 1];
#pragma unroll
            for (int i = 0; i < 16 / Rl; i++)
#pragma unroll
                for (int r = 0; r < Rl; r++) {
                    const int x = b + i * TPL + r * (N / Rl);
                    const float va = v[0][i * Rl + r].x, vb = -v[0][i * Rl + r].y;
                    if (ra) ca[x] = va;
                    if (rb) ca[n + x] = vb;
                    if (__float_as_uint(fabsf(va)) == Ma) {
                        if (va == fabsf(va)) atomicMin(&s_pos[2 * line], x);
                        else atomicMax(&s_neg[2 * line], x);
                    }
                    if (__float_as_uint(fabsf(vb)) == Mb) {
                        if (vb == fabsf(vb)) atomicMin(&s_pos[2 * line + 1], x);
                        else atomicMax(&s_neg[2 * line + 1], x);
                    }
                }
            __syncthreads();
            for (int t = threadIdx.x; t < 2 * G; t += fft::kThreads)
                if (2 * line0 + t < ny)
                    stats[img + 2 * line0 + t] =
                        RowStat{__uint_as_float(s_m[t]), s_pos[t], s_neg[t], 0};
        }
    } else {
        fft::mixed_fill<false>(n, P.dn, G, 0, sm, LS, load);
        const float2 *zs = fft::mixed_transform<1, false>(P, G, 0, sm, sm + G * LS, LS, tw);
        if constexpr (MODE == kRows) {
            fft::mixed_drain<false>(n, P.dn, G, 0, zs, LS, [&](int line, int i, float2 z) {
                const int row = 2 * (line0 + line);
                float *ca = c + (img + row) * n + i;
                if (row < ny) ca[0] = z.x / scale;
                if (row + 1 < ny) ca[n] = -z.y / scale;
            });
        } else {
            // one warp per row: store it and take its statistics
            const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
            const float *sf = reinterpret_cast<const float *>(zs);
            for (int t = warp; t < 2 * G; t += fft::kThreads / 32) {
                const int row = 2 * line0 + t;
                if (row >= ny) continue;
                RowStat s{-1.0f, INT_MAX, -1, 0};
                for (int i = lane; i < n; i += 32) {
                    const float z = sf[2 * ((t >> 1) * LS + pz(i)) + (t & 1)];
                    const float v = t & 1 ? -z : z;
                    c[(img + row) * n + i] = v;
                    s = stat_merge(s, stat_of(v, i));
                }
                s = stat_warp(s);
                if (lane == 0) stats[img + row] = s;
            }
        }
    }
}

// Row statistics of an existing image (for speak on a given correlation map).
__global__ void __launch_bounds__(256) k_row_stats(const float *__restrict__ c, RowStat *stats,
                                                   int nx, int ny) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row = blockIdx.x * 8 + warp, pair = blockIdx.y;
    if (row >= ny) return;
    const float *cr = c + ((size_t)pair * ny + row) * nx;
    RowStat s{-1.0f, INT_MAX, -1, 0};
    for (int i = lane; i < nx; i += 32) s = stat_merge(s, stat_of(cr[i], i));
    s = stat_warp(s);
    if (lane == 0) stats[(size_t)pair * ny + row] = s;
}

// quad2dfit (align2dstack.cpp:1125-1166) in double.
__device__ void quad2dfit_dev(const float *z, float *xsh, float *ysh) {
#define Z(i, j) ((double)z[((j)-1) * 3 + (i)-1])
    const double c2 = (8. * Z(1, 1) - 8. * Z(1, 2) + 5. * Z(2, 1) - 8. * Z(2, 2) + 3. * Z(2, 3) +
                       2. * Z(3, 1) - 8. * Z(3, 2) + 6. * Z(3, 3)) /
                      (-6.);
    const double c3 = (Z(1, 1) - 2. * Z(1, 2) + Z(1, 3) + Z(2, 1) - 2. * Z(2, 2) + Z(2, 3) +
                       Z(3, 1) - 2. * Z(3, 2) + Z(3, 3)) /
                      6.0;
    const double c4 = (8. * Z(1, 1) + 5. * Z(1, 2) + 2. * Z(1, 3) - 8. * Z(2, 1) - 8. * Z(2, 2) -
                       8. * Z(2, 3) + 3. * Z(3, 2) + 6. * Z(3, 3)) /
                      (-6.0);
    const double c5 = (Z(1, 1) - Z(1, 3) - Z(3, 1) + Z(3, 3)) / 4.0;
    const double c6 = (Z(1, 1) + Z(1, 2) + Z(1, 3) - 2. * Z(2, 1) - 2. * Z(2, 2) - 2. * Z(2, 3) +
                       Z(3, 1) + Z(3, 2) + Z(3, 3)) /
                      6.0;
#undef Z
    float ys = 0.0f, xs = 0.0f;
    const double den = 4. * c3 * c6 - c5 * c5;
    if (den != 0.0) {
        ys = (float)((c4 * c5 - 2. * c2 * c6) / den - 2.0);
        xs = (float)((c2 * c5 - 2. * c4 * c3) / den - 2.0);
        if (ys < -1.0f) ys = -1.0f;
        if (ys > 1.0f) ys = 1.0f;
        if (xs < -1.0f) xs = -1.0f;
        if (xs > 1.0f) xs = 1.0f;
    }
    *xsh = xs;
    *ysh = ys;
}

// Pass 4: the reference's peak (speak, align2dstack.cpp:1072-1079) scans x
// outer, y inner, replacing the peak when |v| > pmax and then storing the
// SIGNED v.  Hence: if +M (M = max|v|) occurs, the answer is its first
// occurrence in that order; otherwise the scan passes the last -M and, with
// pmax negative, continues from the next element; that rare case is replayed
// element by element (bounded by the image size).
__global__ void __launch_bounds__(256) k_peak(const float *__restrict__ c,
                                              const RowStat *__restrict__ stats, int nx, int ny,
                                              float *sx, float *sy, int *ixo, int *iyo) {
    __shared__ float sm_m[256];
    __shared__ long long sm_pos[256], sm_neg[256];
    const int pair = blockIdx.x;
    const RowStat *st = stats + (size_t)pair * ny;
    const float *cp = c + (size_t)pair * nx * ny;
    float m = -1.0f;
    for (int r = threadIdx.x; r < ny; r += 256) m = fmaxf(m, st[r].m);
    sm_m[threadIdx.x] = m;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) sm_m[threadIdx.x] = fmaxf(sm_m[threadIdx.x], sm_m[threadIdx.x + o]);
        __syncthreads();
    }
    const float M = sm_m[0];
    // order key in x-major scan order: x * ny + y
    long long pos = LLONG_MAX, neg = -1;
    for (int r = threadIdx.x; r < ny; r += 256) {
        const RowStat s = st[r];
        if (s.m == M) {
            if (s.xpos != INT_MAX) pos = min(pos, (long long)s.xpos * ny + r);
            if (s.xneg >= 0) neg = max(neg, (long long)s.xneg * ny + r);
        }
    }
    sm_pos[threadIdx.x] = pos;
    sm_neg[threadIdx.x] = neg;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) {
            sm_pos[threadIdx.x] = min(sm_pos[threadIdx.x], sm_pos[threadIdx.x + o]);
            sm_neg[threadIdx.x] = max(sm_neg[threadIdx.x], sm_neg[threadIdx.x + o]);
        }
        __syncthreads();
    }
    if (threadIdx.x != 0) return;
    long long t;
    if (!(M > 0.0f)) {
        t = 0;  // nothing exceeds pmax = 0 (the reference leaves the peak undefined)
    } else if (sm_pos[0] != LLONG_MAX) {
        t = sm_pos[0];
    } else {
        // replay the reference's state machine after the last -M
        t = sm_neg[0];
        float pmax = -M;
        const long long n = (long long)nx * ny;
        for (long long u = t + 1; u < n; u++) {
            const int xx = (int)(u / ny), yy = (int)(u % ny);
            const float v = cp[(size_t)yy * nx + xx];
            if (fabsf(v) > pmax) {
                pmax = v;
                t = u;
            }
        }
    }
    const int ix = (int)(t / ny), iy = (int)(t % ny);  // 0-based
    float z[9];
    for (int j = -1; j <= 1; j++)
        for (int i = -1; i <= 1; i++) {
            const int xc = (ix + i + nx) % nx, yc = (iy + j + ny) % ny;
            z[(j + 1) * 3 + (i + 1)] = cp[(size_t)yc * nx + xc];
        }
    float xsh, ysh;
    quad2dfit_dev(z, &xsh, &ysh);
    float xt = xsh + (float)ix, yt = ysh + (float)iy;
    if (xt > (float)(nx / 2)) xt = xt - (float)nx;
    if (yt > (float)(ny / 2)) yt = yt - (float)ny;
    sx[pair] = xt;
    sy[pair] = yt;
    if (ixo) ixo[pair] = ix;
    if (iyo) iyo[pair] = iy;
}

// ---------------------------------------------------------------------------
// Fourier shift (fshift2d) of a stack of images:
//   out = Re(IDFT2(DFT2(in) * exp(i * phase))) / (nx * ny),
//   phase = -2 pi (sx kx + sy ky), frequencies -1/2 at an even length's middle.
// The images are real, so the half spectrum H = nx/2+1 carries everything;
// keeping only the real part of the result is the factor's Hermitian part:
// the factor itself except at the middle frequencies of even lengths, where
// the reference's factor is not conjugate symmetric and its average with the
// conjugate at the mirrored frequency stands in.  The factor is a product
// ex[kx] ey[ky]: one table per image, each entry from an exactly reduced
// argument (the reference rounds the whole phase to float).

// ex[0..H), ey[0..ny) of every image: exp(-2 pi i s k / n).
__global__ void k_fs_phase(const float *__restrict__ sxs, const float *__restrict__ sys, int nx,
                           int ny, float2 *__restrict__ tab) {
    const int H = nx / 2 + 1, i = blockIdx.x * blockDim.x + threadIdx.x, z = blockIdx.y;
    if (i >= H + ny) return;
    const int n = i < H ? nx : ny, j = i < H ? i : i - H;
    const float s = i < H ? sxs[z] : sys[z];
    const float k = (float)(j < (n + 1) / 2 ? j : j - n);
    // s k / n modulo 1: s k as an exact float pair, whole turns taken off exactly
    const float p = __fmul_rn(s, k), pe = __fmaf_rn(s, k, -p);
    const float r = __fadd_rn(__fmaf_rn(-rintf(p / (float)n), (float)n, p), pe);
    float sn, cs;
    sincospif(-2.f * (r / (float)n), &sn, &cs);
    tab[(size_t)z * (H + ny) + i] = make_float2(cs, sn);
}

__device__ __forceinline__ float2 fs_apply(float2 f, float2 ex, float2 ey, bool mx, bool my) {
    float2 e = fft::cmul(ex, ey);
    if (mx || my) {
        if (mx && my) e.y = 0.f;
        else if (mx) e = make_float2(ex.x * ey.x, ex.x * ey.y);
        else e = make_float2(ex.x * ey.x, ex.y * ey.x);
    }
    const float2 g = fft::cmul(f, e);
    return make_float2(g.x, -g.y);  // conjugated: IDFT = conj(DFT(conj))
}

// Column pass of the Fourier shift, in place on F: transforms, the phase
// factor, inverse transforms.
template <int N>
__global__ void __launch_bounds__(fft::kThreads, 3)
    k_fs_cols(float2 *__restrict__ F, int nx, int ny, int ct, int lg, Passes P,
              const float2 *__restrict__ tab, const float2 *__restrict__ tw,
              const float2 *__restrict__ twr) {
    extern __shared__ float4 sm4[];
    float2 *sm = reinterpret_cast<float2 *>(sm4);
    const int n = N > 0 ? N : ny, H = nx / 2 + 1;
    const int c0 = blockIdx.x * ct, LS = col_stride(n, ct, 8);
    const size_t img = (size_t)blockIdx.y * n;
    const float2 *ex = tab + (size_t)blockIdx.y * (H + n) + c0, *ey = ex - c0 + H;
    auto load = [&](int c, int row) -> float2 {
        return c0 + c < H ? F[(img + row) * H + c0 + c] : make_float2(0.f, 0.f);
    };
    auto shift = [&](float2 f, int c, int row) -> float2 {
        if (c0 + c >= H) return f;
        return fs_apply(f, __ldg(ex + c), __ldg(ey + row), 2 * (c0 + c) == nx, 2 * row == n);
    };
    if constexpr (N > 0) {
        using L2 = Pow2<N>;
        constexpr int TPL = L2::TPL, CT = L2::G;
        constexpr int Ra = L2::template radix<false>(0), Rl = L2::template radix<false>(L2::P - 1);
        const int c = threadIdx.x % CT, b = threadIdx.x / CT;
        float2 v[1][16];
#pragma unroll
        for (int i = 0; i < 16 / Ra; i++)
#pragma unroll
            for (int r = 0; r < Ra; r++) v[0][i * Ra + r] = load(c, b + i * TPL + r * (N / Ra));
        fft::transform<N, false, false, 1>(v, sm + c * LS, b, tw);
#pragma unroll
        for (int i = 0; i < 16 / Rl; i++)
#pragma unroll
            for (int r = 0; r < Rl; r++)
                v[0][i * Rl + r] = shift(v[0][i * Rl + r], c, b + i * TPL + r * (N / Rl));
        fft::transform<N, true, false, 1>(v, sm + c * LS, b, twr);
        if (c0 + c >= H) return;
#pragma unroll
        for (int i = 0; i < 16 / Ra; i++)
#pragma unroll
            for (int r = 0; r < Ra; r++) {
                const float2 z = v[0][i * Ra + r];
                F[(img + b + i * TPL + r * (N / Ra)) * H + c0 + c] = make_float2(z.x, -z.y);
            }
    } else {
        fft::mixed_fill<true>(n, P.dn, ct, lg, sm, LS, load);
        float2 *a = sm, *bo = sm + ct * LS;
        for (int pass = 0; pass < 2; pass++) {
            float2 *z = fft::mixed_transform<1, true>(P, ct, lg, a, bo, LS, tw);
            bo = z == a ? bo : a;
            a = z;
            if (pass == 1) break;
            for (int t = threadIdx.x; t < ct * n; t += fft::kThreads) {
                float2 &f = a[(t & (ct - 1)) * LS + pz(t >> lg)];
                f = shift(f, t & (ct - 1), t >> lg);
            }
            __syncthreads();
        }
        fft::mixed_drain<true>(n, P.dn, ct, lg, a, LS, [&](int c, int i, float2 z) {
            if (c0 + c < H) F[(img + i) * H + c0 + c] = make_float2(z.x, -z.y);
        });
    }
}

// ---------------------------------------------------------------------------
// Host side.

// Radices of a length's passes, in order: the kernels' own for powers of two
// from 16, else the fewest out of {2..10, 16} (the smallest sum among those),
// largest first.
static void radices(int n, std::vector<int> &out) {
    out.clear();
    if (n >= 16 && (n & (n - 1)) == 0) {
        const int r0 = n == 512 ? 8 : 16, r1 = n == 512 ? 8 : std::min(16, n / r0);
        for (int r : {r0, r1, n / (r0 * r1)})
            if (r > 1) out.push_back(r);
        return;
    }
    std::vector<int> cur, best;
    int best_sum = INT_MAX;
    auto rec = [&](auto &&self, int m, int top, int sum) -> void {
        if (m == 1) {
            if (best.empty() || cur.size() < best.size() ||
                (cur.size() == best.size() && sum < best_sum)) {
                best = cur;
                best_sum = sum;
            }
            return;
        }
        if (!best.empty() && cur.size() >= best.size()) return;
        for (int r : {16, 10, 9, 8, 7, 6, 5, 4, 3, 2})
            if (r <= top && m % r == 0) {
                cur.push_back(r);
                self(self, m / r, r, sum + r);
                cur.pop_back();
            }
    };
    rec(rec, n, 16, 0);
    out = best;
}

static Passes make_passes(int n, const std::vector<int> &r) {
    Passes p{};
    p.n = n;
    p.np = (int)r.size();
    p.dn = fft::make_fastdiv(n);
    int ns = 1;
    for (int i = 0; i < p.np; i++) {
        p.r[i] = r[i];
        p.ns[i] = ns;
        p.dnr[i] = fft::make_fastdiv(n / r[i]);
        p.dns[i] = fft::make_fastdiv(ns);
        ns *= r[i];
    }
    return p;
}

// Twiddles of both orders of a length's passes (forward at 0, reversed at n).
static void fill_twiddles(int n, float2 *h) {
    std::vector<int> r;
    radices(n, r);
    for (int o = 0; o < 2; o++) {
        int ns = 1;
        for (int R : r) {
            for (int q = 1; q < R; q++)
                for (int k = 0; k < ns; k++) {
                    const double a = 2.0 * M_PI * (double)q * (double)k / ((double)ns * R);
                    h[o * n + ns - 1 + (q - 1) * ns + k] =
                        make_float2((float)std::cos(a), (float)-std::sin(a));
                }
            ns *= R;
        }
        std::reverse(r.begin(), r.end());
    }
}

// A length's passes and its device table (twiddles of both orders).
struct LinePlan {
    Passes fwd;
    const float2 *tw, *twr;
};

static std::mutex g_tw_mu;
static std::map<std::pair<int, int>, float2 *> g_tw;  // (device, N) -> table

static void line_passes(int n, LinePlan *lp) {
    std::vector<int> r;
    radices(n, r);
    lp->fwd = make_passes(n, r);
}

static int line_plan(int N, LinePlan *lp) {
    line_passes(N, lp);
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(g_tw_mu);
    auto it = g_tw.find({dev, N});
    if (it == g_tw.end()) {
        std::vector<float2> h(2 * N, make_float2(0.f, 0.f));
        fill_twiddles(N, h.data());
        float2 *d = nullptr;
        ARECGB_CUDA(dev_malloc(&d, sizeof(float2) * 2 * N));
        cudaError_t e = cudaMemcpy(d, h.data(), sizeof(float2) * 2 * N, cudaMemcpyHostToDevice);
        if (e != cudaSuccess) {
            cudaFree(d);
            ARECGB_CUDA(e);
        }
        it = g_tw.insert({{dev, N}, d}).first;
    }
    lp->tw = it->second;
    lp->twr = it->second + N;
    return 0;
}

// Scratch of the calls below.  It comes from a pool per device that keeps up to
// kPoolBytes between calls: cudaMalloc and cudaFree of 256 MB took a third of a shift
// search on 30 pairs of 750 x 1000 (0.84 ms, 0.59 with the pool).  The pool hands memory
// out in stream order, to any thread and stream; what a call holds beyond the limit
// goes back when its stream is waited for, the rest when a plan is created or an
// allocation of the library fails (scratch_trim).  A capturing stream gets cudaMalloc's
// refusal, as before.
constexpr size_t kPoolBytes = (size_t)512 << 20;
static std::mutex g_pool_mu;
static std::map<int, cudaMemPool_t> g_pool;

static cudaMemPool_t scratch_pool() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
    std::lock_guard<std::mutex> lk(g_pool_mu);
    auto it = g_pool.find(dev);
    if (it != g_pool.end()) return it->second;
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    unsigned long long keep = kPoolBytes;
    if (cudaMemPoolCreate(&pool, &props) != cudaSuccess ||
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
        cudaGetLastError();  // not sticky: cudaMalloc instead
        if (pool) cudaMemPoolDestroy(pool);
        pool = nullptr;
    }
    g_pool[dev] = pool;
    return pool;
}

// Gives the current device's unused scratch back.
void scratch_trim() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return;
    std::lock_guard<std::mutex> lk(g_pool_mu);
    auto it = g_pool.find(dev);
    if (it != g_pool.end() && it->second && cudaMemPoolTrimTo(it->second, 0) != cudaSuccess)
        cudaGetLastError();
}

struct Scratch {
    void *p = nullptr;
    cudaStream_t st = nullptr;
    bool pooled = false;

    int alloc(size_t bytes, cudaStream_t stream) {
        st = stream;
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        const bool known = cudaStreamIsCapturing(st, &cap) == cudaSuccess;
        if (!known) cudaGetLastError();
        cudaMemPool_t pool = known && cap == cudaStreamCaptureStatusNone ? scratch_pool() : nullptr;
        if (pool) {
            pooled = cudaMallocFromPoolAsync(&p, bytes, pool, st) == cudaSuccess;
            if (pooled) return 0;
            cudaGetLastError();
            p = nullptr;
        }
        ARECGB_CUDA(dev_malloc(&p, bytes));
        return 0;
    }
    // Waits for the stream, as the calls do before they return.
    ~Scratch() {
        if (!p) return;
        if (pooled) cudaFreeAsync(p, st);
        cudaStreamSynchronize(st);
        if (!pooled) cudaFree(p);
    }
};

// Calls f with the length as a compile-time constant (0: not a power of two
// from 16).
template <typename F>
static int with_length(int n, F &&f) {
    switch (n) {
#define ARECGB_LEN(n) \
    case n: return f(std::integral_constant<int, n>{});
        ARECGB_LEN(16) ARECGB_LEN(32) ARECGB_LEN(64) ARECGB_LEN(128) ARECGB_LEN(256)
        ARECGB_LEN(512) ARECGB_LEN(1024) ARECGB_LEN(2048) ARECGB_LEN(4096)
#undef ARECGB_LEN
        default: return f(std::integral_constant<int, 0>{});
    }
}

// Forward row pass of nz images (kPairs: image pairs x, y).
template <int MODE>
static int rows_fwd(const LinePlan &lp, const float *x, const float *y, RowSpectra o, int nz,
                    int ny, int nx, cudaStream_t st) {
    return with_length(nx, [&](auto n) -> int {
        auto fn = k_rows_fwd<decltype(n)::value, MODE>;
        const int G = lines_per_block(nx), lines = MODE == kPairs ? ny : (ny + 1) / 2;
        const size_t smem = sizeof(float2) * (size_t)G * plen(nx) * (pow2_length(nx) ? 1 : 2);
        if (int rc = set_smem((const void *)fn, smem)) return rc;
        fn<<<dim3((lines + G - 1) / G, nz), fft::kThreads, smem, st>>>(
            x, y, o, nx, ny, lp.fwd, fft::make_fastdiv(nx / 2 + 1), lp.tw);
        return 0;
    });
}

template <int MODE>
static int rows_inv(const LinePlan &lp, const float2 *W, float *c, RowStat *stats, int nz, int ny,
                    int nx, cudaStream_t st) {
    return with_length(nx, [&](auto n) -> int {
        auto fn = k_rows_inv<decltype(n)::value, MODE>;
        const int G = lines_per_block(nx), lines = (ny + 1) / 2;
        const size_t smem = sizeof(float2) * (size_t)G * plen(nx) * (pow2_length(nx) ? 1 : 2);
        if (int rc = set_smem((const void *)fn, smem)) return rc;
        fn<<<dim3((lines + G - 1) / G, nz), fft::kThreads, smem, st>>>(W, c, stats, nx, ny, lp.fwd,
                                                                      lp.tw);
        return 0;
    });
}

static int log2_of(int n) {
    int l = 0;
    while ((1 << l) < n) l++;
    return l;
}

static int cc_cols(const LinePlan &lp, const float4 *S, float2 *W, int nz, int ny, int nx,
                   cudaStream_t st) {
    return with_length(ny, [&](auto n) -> int {
        auto fn = k_cc_cols<decltype(n)::value>;
        const int ct = col_tile(ny, 16), H = nx / 2 + 1;
        const size_t smem =
            sizeof(float4) * (size_t)ct * col_stride(ny, ct, 16) * (pow2_length(ny) ? 1 : 2);
        if (int rc = set_smem((const void *)fn, smem)) return rc;
        fn<<<dim3((H + ct - 1) / ct, nz), fft::kThreads, smem, st>>>(
            S, W, nx, ny, ct, log2_of(ct), lp.fwd, lp.tw, lp.twr);
        return 0;
    });
}

static int fs_cols(const LinePlan &lp, float2 *F, const float2 *tab, int nz, int ny, int nx,
                   cudaStream_t st) {
    return with_length(ny, [&](auto n) -> int {
        auto fn = k_fs_cols<decltype(n)::value>;
        const int ct = col_tile(ny, 8), H = nx / 2 + 1;
        const size_t smem =
            sizeof(float2) * (size_t)ct * col_stride(ny, ct, 8) * (pow2_length(ny) ? 1 : 2);
        if (int rc = set_smem((const void *)fn, smem)) return rc;
        fn<<<dim3((H + ct - 1) / ct, nz), fft::kThreads, smem, st>>>(
            F, nx, ny, ct, log2_of(ct), lp.fwd, tab, lp.tw, lp.twr);
        return 0;
    });
}

// Scratch of a batch of np pairs, one piece: S [np][ny][H] float4, W
// [np][ny][H] float2.  S is dead once the column pass is done; the
// correlation images and row statistics take its place.
struct CcScratch {
    float4 *S;
    float2 *W;
    float *c;
    RowStat *stats;
};

static size_t round256(size_t b) { return (b + 255) / 256 * 256; }

static size_t cc_s_bytes(int np, int ny, int nx) {
    const size_t spec = (size_t)np * ny * (nx / 2 + 1);
    return round256(sizeof(float4) * spec + 512);  // >= the images and the statistics
}

static size_t cc_bytes(int np, int ny, int nx) {
    return cc_s_bytes(np, ny, nx) + sizeof(float2) * (size_t)np * ny * (nx / 2 + 1);
}

static CcScratch cc_carve(void *p, int np, int ny, int nx) {
    CcScratch s;
    s.S = (float4 *)p;
    s.W = (float2 *)((char *)p + cc_s_bytes(np, ny, nx));
    s.c = (float *)p;
    s.stats = (RowStat *)((char *)p + round256(sizeof(float) * (size_t)np * ny * nx));
    return s;
}

// Correlation images and row statistics of np pairs into s.c and s.stats.
static int correlate_batch(const LinePlan &px, const LinePlan &py, const float *d1,
                           const float *d2, int np, int ny, int nx, const CcScratch &s,
                           cudaStream_t st) {
    int rc = rows_fwd<kPairs>(px, d1, d2, RowSpectra{s.S, nullptr}, np, ny, nx, st);
    if (!rc) rc = cc_cols(py, s.S, s.W, np, ny, nx, st);
    if (!rc) rc = rows_inv<kPairs>(px, s.W, s.c, s.stats, np, ny, nx, st);
    if (!rc) ARECGB_CUDA(cudaGetLastError());
    return rc;
}

// Images per batch: the scratch near `target` bytes.
static int batch_for(int nz, size_t per, size_t target) {
    return (int)std::max<size_t>(
        1, std::min<size_t>(std::min<size_t>((size_t)nz, 65535), target / std::max<size_t>(per, 1)));
}

// Scratch per batch.  Measured on 48 pairs of 2048^2 (50 MB each): 64 MB 3.26
// ms, 128 MB 2.71, 256 MB 2.49, 1 GiB 2.82 — large enough to fill the SMs
// several times over per launch, small enough that part of a batch's spectra
// is still in the 129 MB L2 when the next pass reads it (and to allocate
// quickly).  512^2 images: no difference from 64 MB up.
constexpr size_t kBatchBytes = (size_t)256 << 20;

int cc_shifts(const float *d1, const float *d2, int nz, int ny, int nx, float *sx, float *sy,
              int *ix, int *iy, cudaStream_t st) {
    if (!smooth_length(nx) || !smooth_length(ny) || nz < 0 || !d1 || !d2 || !sx || !sy) {
        set_error("cc_shifts: nx and ny must be in [2, 4096] with prime factors 2, 3, 5, 7 "
                  "(got " + std::to_string(nx) + " x " + std::to_string(ny) + ")");
        return ARECGB_ERR_ARG;
    }
    if (nz == 0) return 0;
    LinePlan px, py;
    int rc = line_plan(nx, &px);
    if (!rc) rc = line_plan(ny, &py);
    if (rc) return rc;
    const int batch = batch_for(nz, cc_bytes(1, ny, nx), kBatchBytes);
    Scratch buf;
    if ((rc = buf.alloc(cc_bytes(batch, ny, nx), st))) return rc;
    for (int p0 = 0; !rc && p0 < nz; p0 += batch) {
        const int np = std::min(batch, nz - p0);
        const size_t off = (size_t)p0 * nx * ny;
        const CcScratch s = cc_carve(buf.p, np, ny, nx);
        rc = correlate_batch(px, py, d1 + off, d2 + off, np, ny, nx, s, st);
        if (rc) break;
        k_peak<<<np, 256, 0, st>>>(s.c, s.stats, nx, ny, sx + p0, sy + p0, ix ? ix + p0 : nullptr,
                                   iy ? iy + p0 : nullptr);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) {
            set_error(std::string("cc_shifts: ") + cudaGetErrorString(e));
            rc = cuda_status(e);
        }
    }
    return rc;
}

int ccorr_image(const float *dx, const float *dy, float *dc, int ny, int nx, cudaStream_t st) {
    if (!smooth_length(nx) || !smooth_length(ny)) {
        set_error("ccorr2d: nx and ny must be in [2, 4096] with prime factors 2, 3, 5, 7 (got " +
                  std::to_string(nx) + " x " + std::to_string(ny) + ")");
        return ARECGB_ERR_ARG;
    }
    LinePlan px, py;
    int rc = line_plan(nx, &px);
    if (!rc) rc = line_plan(ny, &py);
    if (rc) return rc;
    Scratch buf;
    if ((rc = buf.alloc(cc_bytes(1, ny, nx), st))) return rc;
    CcScratch s = cc_carve(buf.p, 1, ny, nx);
    s.c = dc;
    rc = correlate_batch(px, py, dx, dy, 1, ny, nx, s, st);
    return rc;
}

int fshift_stack(const float *d_in, float *d_out, int nz, int ny, int nx, const float *d_sx,
                 const float *d_sy, cudaStream_t st) {
    if (!smooth_length(nx) || !smooth_length(ny) || ny > 2048 || nz < 0 || !d_in || !d_out ||
        !d_sx || !d_sy) {
        set_error("fshift2d: nx in [2, 4096] and ny in [2, 2048] with prime factors 2, 3, 5, 7 "
                  "(got " + std::to_string(nx) + " x " + std::to_string(ny) + ")");
        return ARECGB_ERR_ARG;
    }
    if (nz == 0) return 0;
    LinePlan px, py;
    int rc = line_plan(nx, &px);
    if (!rc) rc = line_plan(ny, &py);
    if (rc) return rc;
    const int H = nx / 2 + 1;
    const size_t spec = sizeof(float2) * (size_t)ny * H, tabs = sizeof(float2) * (size_t)(H + ny);
    const int batch = batch_for(nz, spec + tabs, kBatchBytes);
    Scratch buf;
    if ((rc = buf.alloc((spec + tabs) * batch, st))) return rc;
    float2 *F = (float2 *)buf.p, *tab = F + (size_t)ny * H * batch;
    for (int z0 = 0; z0 < nz && !rc; z0 += batch) {
        const int nb = std::min(batch, nz - z0);
        const size_t off = (size_t)z0 * nx * ny;
        k_fs_phase<<<dim3((H + ny + 127) / 128, nb), 128, 0, st>>>(d_sx + z0, d_sy + z0, nx, ny, tab);
        rc = rows_fwd<kRows>(px, d_in + off, nullptr, RowSpectra{nullptr, F}, nb, ny, nx, st);
        if (!rc) rc = fs_cols(py, F, tab, nb, ny, nx, st);
        if (!rc) rc = rows_inv<kRows>(px, F, d_out + off, nullptr, nb, ny, nx, st);
        count_launches(4);
        cudaError_t e = cudaGetLastError();
        if (!rc && e != cudaSuccess) {
            set_error(std::string("fshift2d: ") + cudaGetErrorString(e));
            rc = cuda_status(e);
        }
    }
    return rc;
}

int peak_search(const float *dc, int nz, int ny, int nx, float *sx, float *sy, int *ix, int *iy,
                cudaStream_t st) {
    if (nx < 1 || ny < 1 || nz < 1) {
        set_error("speak: bad shape");
        return ARECGB_ERR_ARG;
    }
    Scratch buf;
    if (int rc = buf.alloc(sizeof(RowStat) * (size_t)ny * nz, st)) return rc;
    RowStat *stats = (RowStat *)buf.p;
    k_row_stats<<<dim3((ny + 7) / 8, nz), 256, 0, st>>>(dc, stats, nx, ny);
    k_peak<<<nz, 256, 0, st>>>(dc, stats, nx, ny, sx, sy, ix, iy);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error(std::string("speak: ") + cudaGetErrorString(e));
        return cuda_status(e);
    }
    return 0;
}
// ---------------------------------------------------------------------------
// Shift search without allocation (arecgb_cc_shifts_static).
//
// For callers that must not allocate device memory while they run: an
// alignment loop that interleaves shift searches with a reconstruction running
// on another stream (cc_shifts waits for its own stream before it returns, and for the
// whole device where its pool cannot serve it and cudaFree takes its place), or a
// host whose memory is owned by another allocator (a caching allocator that already
// holds the free HBM).
//
// Scratch: one file-scope device array of kStaticBytes (3.5 MiB), carved into
//   S       float4 [kStaticSpec]   half spectra of both images; then the
//                                  correlation images and row statistics
//   W       float2 [kStaticSpec]   the product's spectrum after the column pass
//   tw      float2 [2016]          twiddles for N = 16..512, both pass orders,
//                                  table N at offset 2 (N - 16)
// Limit: nx, ny powers of two in [16, 512] and nz * ny * nx <= kStaticPixels
// (one 512 x 512 pair, or e.g. 64 pairs of 64 x 64).  Larger requests are
// rejected with ARECGB_ERR_ARG; arecgb_cc_shifts has no such limit.
// Nothing in the scratch must start at zero: every element a call reads was
// written earlier in the same call (row pass -> column pass -> inverse rows ->
// peak).  Only the twiddle tables persist; the set-up writes them.
// The scratch is shared by every call on a device: two calls that can overlap
// (different streams, or host threads without ordering) race on it.
constexpr size_t kStaticPixels = 512 * 512;
constexpr size_t kStaticRows = kStaticPixels / 16;                  // ny * nz <= pixels / nx
constexpr size_t kStaticSpec = kStaticPixels / 2 + kStaticRows;     // (nx/2 + 1) * ny * nz
constexpr size_t kStaticTw = 2048;                                  // 2 (16 + ... + 512) = 2016
constexpr size_t kOffW = (sizeof(float4) * kStaticSpec + 512 + 255) / 256 * 256;
constexpr size_t kOffTw = kOffW + sizeof(float2) * kStaticSpec;
constexpr size_t kStaticBytes = kOffTw + sizeof(float2) * kStaticTw;
static_assert(kOffW % 256 == 0 && kOffTw % 256 == 0, "scratch pieces must stay 256-byte aligned");

static __device__ __align__(256) unsigned char g_cc_static[kStaticBytes];

struct StaticScratch {
    bool ready = false;
    unsigned char *base = nullptr;
};
static std::mutex g_static_mu;
static std::map<int, StaticScratch> g_static;  // device -> scratch address

// Once per device, with that device current: resolve the scratch address and
// write the twiddle tables (a synchronous copy).  Run the first call before
// any stream capture.
static int static_setup(unsigned char **base) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        set_error(std::string("cc_shifts_static: cudaGetDevice: ") + cudaGetErrorString(e));
        return cuda_status(e);
    }
    std::lock_guard<std::mutex> lk(g_static_mu);
    StaticScratch &s = g_static[dev];
    if (s.ready) {
        *base = s.base;
        return 0;
    }
    void *ptr = nullptr;
    e = cudaGetSymbolAddress(&ptr, g_cc_static);
    if (e != cudaSuccess || !ptr) {
        set_error(std::string("cc_shifts_static: cudaGetSymbolAddress: ") +
                  cudaGetErrorString(e));
        return cuda_status(e != cudaSuccess ? e : cudaErrorInvalidSymbol);
    }
    std::vector<float2> h(kStaticTw, make_float2(0.f, 0.f));
    for (int N = 16; N <= 512; N *= 2) fill_twiddles(N, h.data() + 2 * (N - 16));
    e = cudaMemcpy((unsigned char *)ptr + kOffTw, h.data(), sizeof(float2) * kStaticTw,
                   cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        set_error(std::string("cc_shifts_static: twiddle upload: ") + cudaGetErrorString(e));
        return cuda_status(e);
    }
    s.base = (unsigned char *)ptr;
    s.ready = true;
    *base = s.base;
    return 0;
}

int cc_shifts_static(const float *d1, const float *d2, int nz, int ny, int nx, float *sx,
                     float *sy, int *ix, int *iy, cudaStream_t st) {
    const bool shape_ok = nx >= 16 && nx <= 512 && ny >= 16 && ny <= 512 &&
                          (nx & (nx - 1)) == 0 && (ny & (ny - 1)) == 0;
    if (!shape_ok || nz < 0 || !d1 || !d2 || !sx || !sy) {
        set_error("cc_shifts_static: nx and ny must be powers of two in [16, 512]");
        return ARECGB_ERR_ARG;
    }
    if ((size_t)nz * ny * nx > kStaticPixels) {
        set_error("cc_shifts_static: nz * ny * nx = " + std::to_string((size_t)nz * ny * nx) +
                  " exceeds the static scratch limit of " + std::to_string(kStaticPixels) +
                  " pixels (one 512 x 512 pair); use arecgb_cc_shifts");
        return ARECGB_ERR_ARG;
    }
    unsigned char *base = nullptr;
    int rc = static_setup(&base);
    if (rc) return rc;
    if (nz == 0) return 0;
    const float2 *tw = reinterpret_cast<const float2 *>(base + kOffTw);
    LinePlan px, py;
    line_passes(nx, &px);
    line_passes(ny, &py);
    px.tw = tw + 2 * (nx - 16);
    px.twr = px.tw + nx;
    py.tw = tw + 2 * (ny - 16);
    py.twr = py.tw + ny;
    // nz ny (nx/2 + 1) <= kStaticSpec for every accepted shape, so S and W end
    // before the twiddles
    const CcScratch s = cc_carve(base, nz, ny, nx);
    if ((rc = correlate_batch(px, py, d1, d2, nz, ny, nx, s, st))) return rc;
    k_peak<<<nz, 256, 0, st>>>(s.c, s.stats, nx, ny, sx, sy, ix, iy);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error(std::string("cc_shifts_static: ") + cudaGetErrorString(e));
        return cuda_status(e);
    }
    return 0;
}

}  // namespace arecgb

extern "C" int arecgb_cc_shifts_static(const float *d_img1, const float *d_img2, int nz, int ny,
                                       int nx, float *d_sx, float *d_sy, int *d_ix, int *d_iy,
                                       void *stream) {
    return arecgb::cc_shifts_static(d_img1, d_img2, nz, ny, nx, d_sx, d_sy, d_ix, d_iy,
                                    (cudaStream_t)stream);
}
