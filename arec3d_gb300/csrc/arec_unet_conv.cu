// 3x3 convolution (stride 1, zero padding 1) as an implicit GEMM on the
// 5th-generation tensor cores: tcgen05.mma (BF16 x BF16 -> FP32 in TMEM).
//
//   Y[p][co] = act( bias[co] + sum_{tap, ci} X[p + tap][ci] * Wt[co][tap][ci] )
//
// X, Y: NHWC bf16 ([P = n*H*W pixels][C]); Wt: [Cout][9][Cin] bf16.
// A block owns 128 consecutive pixels (GEMM M = 128) and all Cout output
// channels (GEMM N = Cout in {32, 64, 128, 256}); K = 9*Cin runs in chunks of
// 32 channels of one tap.  Per chunk, 128 threads gather the A slab (the 128
// pixels' shifted neighbours, zeros outside the image) and the B slab (weights)
// into shared memory in the tensor core's K-major layout; one thread issues two
// tcgen05.mma (K = 16 each) into the TMEM accumulator and commits them to the
// stage's mbarrier, so the next chunk's gather overlaps the MMAs (two stages).
// The epilogue reads TMEM with tcgen05.ld (warp w: pixels 32w..32w+31), adds
// the bias, applies ReLU and stores bf16.
//
// The same kernel computes the data gradient of a convolution from the
// spatially flipped, channel-transposed weights.
#include <cuda.h>  // CUtensorMap and its enums (the encoder comes from the runtime's entry point)
#include <cuda_bf16.h>
#include <stdint.h>

#include <mutex>

#include "arec_internal.cuh"
#include "arec_umma.cuh"

namespace arecgb {

constexpr int kConvKC = 32;          // input channels per K chunk
constexpr uint32_t kWaitLimit = 4u << 20;

template <int COUT>
struct ConvCfg {
    static constexpr int A_BYTES = 128 * kConvKC * 2;  // 8 KB
    static constexpr int B_BYTES = COUT * kConvKC * 2;
    static constexpr int STAGE = A_BYTES + B_BYTES;
    static constexpr int SMEM = 2 * STAGE;
    static constexpr uint32_t NCOLS = COUT < 32 ? 32 : COUT;
};

// byte offset of element (row, k) (k < 32) in a K-major no-swizzle slab with
// `rows` rows: two MMA slabs (K = 16 each) of rows/8 core-matrix groups.
__device__ __forceinline__ int kmaj_offset(int row, int kpiece /*0..3, 8 elements*/, int rows) {
    const int s = kpiece >> 1, j = kpiece & 1;
    return s * (rows / 8) * 256 + (row >> 3) * 256 + j * 128 + (row & 7) * 16;
}

template <int COUT, int LBO, int SBO>
__global__ void __launch_bounds__(128)
    conv3x3_umma_kernel(const __nv_bfloat16 *__restrict__ X, const __nv_bfloat16 *__restrict__ Wt,
                        const float *__restrict__ bias, __nv_bfloat16 *__restrict__ Y, int H,
                        int Wd, int Cin, int P, int relu, int ystride, int *err) {
    using Cfg = ConvCfg<COUT>;
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ uint64_t mbar[2];
    __shared__ uint32_t tmem_base;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int p0 = blockIdx.x * 128;

    if (warp == 0) {
        umma::tmem_alloc(&tmem_base, Cfg::NCOLS);
        umma::tmem_relinquish();
    }
    if (tid == 0) {
        umma::mbar_init(&mbar[0], 1);
        umma::mbar_init(&mbar[1], 1);
        umma::mbar_fence_init();
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = tmem_base;

    // this thread's pixel (row of A)
    const int p = p0 + tid;
    const bool pvalid = p < P;
    const int hw = H * Wd;
    const int n = p / hw, h = (p / Wd) % H, w = p % Wd;
    const int cchunks = Cin / kConvKC;
    const int nchunks = 9 * cchunks;
    constexpr uint32_t idesc = umma::idesc_bf16(128, COUT);
    bool ok = true;

    for (int c = 0; c < nchunks; c++) {
        const int st = c & 1;
        if (c >= 2 && ok) {
            if (!umma::mbar_wait(&mbar[st], ((c - 2) >> 1) & 1, kWaitLimit)) ok = false;
        }
        unsigned char *A = sm + st * Cfg::STAGE;
        unsigned char *B = A + Cfg::A_BYTES;
        const int tap = c / cchunks, c0 = (c % cchunks) * kConvKC;
        const int dy = tap / 3 - 1, dx = tap % 3 - 1;
        // A: pixel tid, its neighbour at (dy, dx), channels c0..c0+31 (4 x 16 B)
        {
            const int hh = h + dy, ww = w + dx;
            const bool inside = pvalid && hh >= 0 && hh < H && ww >= 0 && ww < Wd;
            const uint4 *src = reinterpret_cast<const uint4 *>(
                X + ((size_t)n * hw + (size_t)(inside ? hh : 0) * Wd + (inside ? ww : 0)) * Cin + c0);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                uint4 v = inside ? __ldg(src + q) : make_uint4(0, 0, 0, 0);
                *reinterpret_cast<uint4 *>(A + kmaj_offset(tid, q, 128)) = v;
            }
        }
        // B: weights Wt[co][tap][c0..c0+31]
        for (int i = tid; i < COUT * 4; i += 128) {
            const int co = i >> 2, q = i & 3;
            const uint4 v = __ldg(reinterpret_cast<const uint4 *>(
                Wt + ((size_t)co * 9 + tap) * Cin + c0 + q * 8));
            *reinterpret_cast<uint4 *>(B + kmaj_offset(co, q, COUT)) = v;
        }
        umma::fence_async_smem();
        umma::fence_before_sync();
        __syncthreads();
        umma::fence_after_sync();
        if (tid == 0 && ok) {
#pragma unroll
            for (int s = 0; s < 2; s++) {
                const uint64_t ad = umma::smem_desc(umma::smem_addr(A + s * (128 / 8) * 256), LBO, SBO);
                const uint64_t bd =
                    umma::smem_desc(umma::smem_addr(B + s * (COUT / 8) * 256), LBO, SBO);
                umma::mma_bf16(tmem, ad, bd, idesc, (c > 0 || s > 0) ? 1u : 0u);
            }
            umma::mma_commit(&mbar[st]);
        }
    }
    // all MMAs done (the last commit covers every earlier MMA of the issuing thread)
    if (nchunks > 0 && ok) {
        const int last = nchunks - 1;
        if (!umma::mbar_wait(&mbar[last & 1], (last >> 1) & 1, kWaitLimit)) ok = false;
    }
    if (!ok && lane == 0) atomicOr(err, 4);
    umma::fence_after_sync();

    // epilogue: warp w reads TMEM lanes 32w.. (pixels p0 + 32w + lane)
    if (ok) {
#pragma unroll 1
        for (int cc = 0; cc < COUT / 32; cc++) {
            float v[32];
            umma::tmem_ld32(tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)(cc * 32), v);
            if (pvalid) {
                __align__(16) __nv_bfloat16 out[32];
#pragma unroll
                for (int i = 0; i < 32; i++) {
                    float t = v[i] + (bias ? bias[cc * 32 + i] : 0.f);
                    if (relu) t = fmaxf(t, 0.f);
                    out[i] = __float2bfloat16(t);
                }
                uint4 *dst = reinterpret_cast<uint4 *>(Y + (size_t)p * ystride + cc * 32);
#pragma unroll
                for (int q = 0; q < 4; q++) dst[q] = reinterpret_cast<const uint4 *>(out)[q];
            }
        }
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) umma::tmem_dealloc(tmem, Cfg::NCOLS);
}

template <int COUT, int LBO, int SBO>
static int launch_conv(const __nv_bfloat16 *X, const __nv_bfloat16 *Wt, const float *bias,
                       __nv_bfloat16 *Y, int H, int Wd, int Cin, int P, int relu, int ystride,
                       int *err, cudaStream_t st) {
    using Cfg = ConvCfg<COUT>;
    if (int rc = set_smem((const void *)conv3x3_umma_kernel<COUT, LBO, SBO>, Cfg::SMEM)) return rc;
    conv3x3_umma_kernel<COUT, LBO, SBO><<<(P + 127) / 128, 128, Cfg::SMEM, st>>>(
        X, Wt, bias, Y, H, Wd, Cin, P, relu, ystride, err);
    ARECGB_CUDA(cudaGetLastError());
    return 0;
}

// ---------------------------------------------------------------------------
// TMA path.  One block per SM runs over the layer's tiles; one warp loads (TMA),
// one issues the MMAs, four take the sums from TMEM to global memory, so that a
// tile's loads, products and stores overlap its neighbours'.
//
// A chunk of K is 32 or 64 input channels of one tap (or one column of taps): its
// pixels come from an NHWC tensor map (rows and columns outside the image arrive
// as zeros, which is the convolution's padding), its weights from a
// [Cout][9][Cin] one, both with the 64 or 128-byte swizzle the tensor core reads
// directly.  Two kinds of tiles, which add the same products in different orders:
//
// - BAND (32 or 64 output channels, widths that are multiples of 128): R rows of
//   128 pixels, chunks over (dx, channels).  One box brings the R + 2 input rows,
//   shifted by dx, and three the weights of the taps (dy, dx).  Input row j
//   adds to the output rows j - 2 .. j with the taps dy = 2 .. 0: their sums are
//   neighbouring columns of TMEM and the three weight slabs, in that order, one
//   operand, so one MMA (N = 3 Cout) takes all three: a narrow MMA is bound by
//   the reading of its A operand (44 clocks at N = 32, 56 at 96).  Per output
//   row the order is (dx, channels, dy).
// - otherwise R tiles of 128 pixels (2^lw x 128 / 2^lw, one above the other),
//   chunks over (tap, channels); the tiles share a chunk's weights.
//
// What bounds it: the loads into shared memory (a band's rows arrive three times, a
// tile's pixels nine times), at most 70 bytes per clock and SM from L2, and half
// of that for rows of 64 bytes: where the input channels allow it a chunk is 64 of
// them (the order of the products stays).  Forward pass at 16 x 1024^2, all layers
// of a kind, from blocks of one tile each with one-lane issue (4.5, 3.0, 2.4 and
// 0.46 ms for 32, 64, 128 and 256 output channels): 2.6, 1.6, 1.9 and 0.45 ms with
// 32-channel chunks, 2.4, 1.6, 1.3 and 0.32 ms with 64.
template <int COUT, int R, bool BAND, int KC, int ST>
struct PipeCfg {
    static constexpr int STAGES = ST;
    static constexpr int A_TILE = 128 * KC * 2;  // 128 pixels
    static constexpr int A_BYTES = (BAND ? R + 2 : R) * A_TILE;
    static constexpr int B_TAP = COUT * KC * 2;  // one tap's weights
    static constexpr int STAGE = A_BYTES + (BAND ? 3 : 1) * B_TAP;  // a multiple of 1024
    static constexpr int OUT = 32 * 64;      // a warp's 32 pixels x 32 channels
    static constexpr int NOUT = STAGES * STAGE > 212 * 1024 ? 1 : 2;  // such buffers per warp
    static constexpr int SMEM = STAGES * STAGE + 4 * NOUT * OUT + 1024;
    static_assert(SMEM <= 227 * 1024 - 1024, "shared memory");
    static constexpr int COLS = R * COUT;
    static constexpr uint32_t NCOLS = 2 * COLS <= 256 ? 2 * COLS : 512;  // two sets of sums
};
// K-major operand whose rows are KC channels: 64-byte or 128-byte swizzle.
template <int KC>
__device__ __forceinline__ uint64_t desc_k(uint32_t saddr) {
    if (KC == 32) return umma::smem_desc_sw64(saddr);
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFF);
    d |= (uint64_t)1 << 16;            // leading byte offset (unused for this layout)
    d |= (uint64_t)(1024 >> 4) << 32;  // stride byte offset
    d |= (uint64_t)1 << 46;            // version
    d |= (uint64_t)2 << 61;            // 128-byte swizzle
    return d;
}

constexpr int kPipeLoad = 4, kPipeMma = 5, kPipeThreads = 32 * 6;

template <int COUT, int R, bool BAND, int KC, int ST>
__global__ void __launch_bounds__(kPipeThreads, 1)
    conv3x3_pipe_kernel(const __grid_constant__ CUtensorMap tmX,
                        const __grid_constant__ CUtensorMap tmW,
                        const __grid_constant__ CUtensorMap tmY, const float *__restrict__ bias, int H,
                        int Wd, int Cin, int lw, int relu, int wt, int ht, int ntiles, int *err) {
    using Cfg = PipeCfg<COUT, R, BAND, KC, ST>;
    static_assert(Cfg::NCOLS >= 32 && 2 * Cfg::COLS <= 512 && (Cfg::NCOLS & (Cfg::NCOLS - 1)) == 0,
                  "TMEM columns: a power of two in [32, 512]");
    static_assert(Cfg::STAGE % 1024 == 0, "stages stay 1024-byte aligned");
    extern __shared__ unsigned char sm_raw[];
    __shared__ __align__(8) uint64_t full[ST], empty[ST], accfull[2], accfree[2], drained;
    __shared__ __align__(16) float s_bias[COUT];
    __shared__ uint32_t tmem_base;
    const uint32_t raw = umma::smem_addr(sm_raw);
    unsigned char *sm = sm_raw + ((1024u - (raw & 1023u)) & 1023u);  // 1024-byte aligned stages
    const int tid = threadIdx.x, warp = umma::uniform(tid >> 5), lane = tid & 31;
    const int cchunks = Cin / KC, nchunks = (BAND ? 3 : 9) * cchunks;
    const int hb = BAND ? R : (128 >> lw) * R;  // image rows per tile

    if (warp == kPipeLoad) {
        umma::tmem_alloc(&tmem_base, Cfg::NCOLS);
        umma::tmem_relinquish();
    }
    if (tid == 0) {
        for (int s = 0; s < ST; s++) {
            umma::mbar_init(&full[s], 1);
            umma::mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; b++) {
            umma::mbar_init(&accfull[b], 1);
            umma::mbar_init(&accfree[b], 4);
        }
        umma::mbar_init(&drained, 1);
        umma::mbar_fence_init();
    }
    for (int i = tid; i < COUT; i += kPipeThreads) s_bias[i] = bias ? bias[i] : 0.f;
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = umma::uniform(tmem_base);

    if (warp == kPipeLoad) {
        if (lane == 0) {
            bool ok = true;
            int it = 0;
            for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
                const int w0 = t % wt << lw, h0 = t / wt % ht * hb, n = t / wt / ht;
                for (int c = 0; c < nchunks; c++, it++) {
                    const int s = it % ST;
                    if (it >= ST &&
                        !umma::mbar_wait(&empty[s], (uint32_t)(it / ST - 1) & 1u, kWaitLimit)) {
                        ok = false;
                        break;
                    }
                    const int tap = c / cchunks, c0 = (c % cchunks) * KC;
                    unsigned char *A = sm + s * Cfg::STAGE, *B = A + Cfg::A_BYTES;
                    umma::mbar_arrive_expect_tx(&full[s], (uint32_t)Cfg::STAGE);
                    if (BAND) {
                        umma::tma_load_4d(A, &tmX, c0, w0 + tap - 1, h0 - 1, n, &full[s]);
#pragma unroll
                        for (int dy = 0; dy < 3; dy++)
                            umma::tma_load_3d(B + (2 - dy) * Cfg::B_TAP, &tmW, c0, 3 * dy + tap, 0,
                                              &full[s]);
                    } else {
                        umma::tma_load_4d(A, &tmX, c0, w0 + tap % 3 - 1, h0 + tap / 3 - 1, n, &full[s]);
                        umma::tma_load_3d(B, &tmW, c0, tap, 0, &full[s]);
                    }
                }
            }
            if (!ok) {
                atomicOr(err, 4);
                umma::ring_drain(full, ST, it, kWaitLimit);
            }
        }
        __syncwarp();
    } else if (warp == kPipeMma) {
        const uint32_t sm0 = umma::uniform(umma::smem_addr(sm));
        bool ok = true;
        int it = 0, i = 0;
        for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x, i++) {
            const uint32_t tm = tmem + (uint32_t)((i & 1) * Cfg::COLS);
            if (i >= 2) ok = umma::mbar_wait_warp(&accfree[i & 1], (uint32_t)(i / 2 - 1) & 1u, kWaitLimit);
            for (int c = 0; c < nchunks && ok; c++, it++) {
                const int s = it % ST;
                ok = umma::mbar_wait_warp(&full[s], (uint32_t)(it / ST) & 1u, kWaitLimit);
                if (!ok) break;
                umma::fence_after_sync();
                const uint32_t a = sm0 + (uint32_t)(s * Cfg::STAGE), bw = a + Cfg::A_BYTES;
                if (BAND) {
#pragma unroll
                    for (int half = 0; half < KC / 32; half++)
#pragma unroll
                        for (int j = 0; j < R + 2; j++) {
                            // output rows r0 .. r1, their taps from slab s0 on
                            const int r0 = j < 2 ? 0 : j - 2, r1 = j < R ? j : R - 1;
                            const int s0 = j < 2 ? 2 - j : 0;
                            const uint32_t d = tm + (uint32_t)(r0 * COUT);
#pragma unroll
                            for (int k = 2 * half; k < 2 * half + 2; k++) {
                                const uint64_t ad = desc_k<KC>(a + j * Cfg::A_TILE + 32 * k);
                                const uint64_t bd = desc_k<KC>(bw + s0 * Cfg::B_TAP + 32 * k);
                                if (c == 0 && k == 0 && j < R) {
                                    // output row j starts here (dy = 0, the last slab)
                                    if (r1 > r0)
                                        umma::mma_f16_warp(d, ad, bd,
                                                           umma::idesc_bf16(128, (r1 - r0) * COUT), 1u);
                                    umma::mma_f16_warp(tm + (uint32_t)(j * COUT), ad,
                                                       desc_k<KC>(bw + 2 * Cfg::B_TAP),
                                                       umma::idesc_bf16(128, COUT), 0u);
                                } else {
                                    umma::mma_f16_warp(d, ad, bd,
                                                       umma::idesc_bf16(128, (r1 - r0 + 1) * COUT), 1u);
                                }
                            }
                        }
                } else {
#pragma unroll
                    for (int m = 0; m < R; m++)
#pragma unroll
                        for (int k = 0; k < KC / 16; k++)
                            umma::mma_f16_warp(tm + (uint32_t)(m * COUT),
                                               desc_k<KC>(a + m * Cfg::A_TILE + 32 * k),
                                               desc_k<KC>(bw + 32 * k), umma::idesc_bf16(128, COUT),
                                               (c > 0 || k > 0) ? 1u : 0u);
                }
                umma::mma_commit_warp(&empty[s]);
            }
            if (ok) umma::mma_commit_warp(&accfull[i & 1]);
        }
        if (!ok) {
            if (lane == 0) atomicOr(err, 4);
            umma::mma_drain_warp(&drained, kWaitLimit);
        }
        __syncwarp();
    } else {
        // TMEM lane = pixel of a tile, this warp's from 32 warp on
        unsigned char *out = sm + ST * Cfg::STAGE + warp * Cfg::NOUT * Cfg::OUT;
        const int pw = (32 * warp) & ((1 << lw) - 1), ph = (32 * warp) >> lw;
        bool ok = true;
        int i = 0, q = 0;
        for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x, i++) {
            const int w0 = (t % wt << lw) + pw, h0 = t / wt % ht * hb + ph, n = t / wt / ht;
            ok = __all_sync(0xffffffffu,
                            umma::mbar_wait(&accfull[i & 1], (uint32_t)(i / 2) & 1u, kWaitLimit));
            if (!ok) break;
            umma::fence_after_sync();
            const uint32_t tm = tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)((i & 1) * Cfg::COLS);
#pragma unroll 1
            for (int cc = 0; cc < Cfg::COLS / 32; cc++) {
                const int m = cc / (COUT / 32), c0 = cc % (COUT / 32) * 32;
                const int h = h0 + (BAND ? m : m * (128 >> lw));
                float v[32];
                umma::tmem_ld32(tm + (uint32_t)(cc * 32), v);
                if (cc == Cfg::COLS / 32 - 1) {
                    umma::fence_before_sync();
                    __syncwarp();
                    if (lane == 0) umma::mbar_arrive(&accfree[i & 1]);
                }
                if (w0 >= Wd || h >= H) continue;  // uniform over the warp
                if (lane == 0) umma::tma_store_wait_read<Cfg::NOUT - 1>();
                __syncwarp();
                const float4 *bs = reinterpret_cast<const float4 *>(s_bias + c0);
#pragma unroll
                for (int g = 0; g < 4; g++) {  // 8 channels, 16 bytes, swizzled as the map has it
                    const float4 b0 = bs[2 * g], b1 = bs[2 * g + 1];
                    const float bb[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
                    __align__(16) __nv_bfloat16 o[8];
#pragma unroll
                    for (int e = 0; e < 8; e++) {
                        float f = v[8 * g + e] + bb[e];
                        if (relu) f = fmaxf(f, 0.f);
                        o[e] = __float2bfloat16(f);
                    }
                    *reinterpret_cast<uint4 *>(out + q * Cfg::OUT + lane * 64 +
                                               ((g ^ ((lane >> 1) & 3)) << 4)) =
                        *reinterpret_cast<const uint4 *>(o);
                }
                umma::fence_async_smem();
                __syncwarp();
                if (lane == 0) umma::tma_store_4d(&tmY, out + q * Cfg::OUT, c0, w0, h, n);
                q = (q + 1) % Cfg::NOUT;
            }
        }
        if (!ok && lane == 0) atomicOr(err, 4);
        if (lane == 0) umma::tma_store_wait_read<0>();
        __syncwarp();
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == kPipeLoad) umma::tmem_dealloc(tmem, Cfg::NCOLS);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                  const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled() {
    static std::once_flag once;
    static EncodeTiledFn fn = nullptr;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                             &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    });
    return fn;
}

bool encode_rows_map(CUtensorMap *m, const float *base, int ys, int nrows, int box_cols,
                     int box_rows) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc) return false;
    const cuuint64_t d[2] = {(cuuint64_t)ys, (cuuint64_t)nrows};
    const cuuint64_t st[1] = {(cuuint64_t)ys * 4};
    const cuuint32_t b[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
    const cuuint32_t one[2] = {1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, (void *)base, d, st, b, one,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
               CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// FP16 pairs [2][n2][n1][ys] (arec_project_mma.cuh): box = 64 slices x box1 x
// box2 of one part, 128-byte swizzle.
bool encode_half_map(CUtensorMap *m, const void *base, int ys, int n1, int n2, int box1, int box2) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc) return false;
    const cuuint64_t d[4] = {(cuuint64_t)ys, (cuuint64_t)n1, (cuuint64_t)n2, 2};
    const cuuint64_t st[3] = {(cuuint64_t)ys * 2, (cuuint64_t)ys * 2 * n1, (cuuint64_t)ys * 2 * n1 * n2};
    const cuuint32_t b[4] = {64, (cuuint32_t)box1, (cuuint32_t)box2, 1};
    const cuuint32_t one[4] = {1, 1, 1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, (void *)base, d, st, b, one,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
               CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// FP16 pairs [2][na][groups][nx][8]: box = box_bins bins of 8 slices x 16 slice
// groups of one angle and part.
bool encode_foot_map(CUtensorMap *m, const void *base, int nx, int groups, int na, int box_bins) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc) return false;
    const cuuint64_t row = (cuuint64_t)nx * 16;
    const cuuint64_t d[4] = {(cuuint64_t)nx * 8, (cuuint64_t)groups, (cuuint64_t)na, 2};
    const cuuint64_t st[3] = {row, row * groups, row * groups * na};
    const cuuint32_t b[4] = {(cuuint32_t)box_bins * 8, 16, 1, 1};
    const cuuint32_t one[4] = {1, 1, 1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, (void *)base, d, st, b, one,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool encode_sino_map(CUtensorMap *m, const float *base, int ys, int nx, int na, int box_cols,
                     int box_bins) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc) return false;
    const cuuint64_t d[3] = {(cuuint64_t)ys, (cuuint64_t)nx, (cuuint64_t)na};
    const cuuint64_t st[2] = {(cuuint64_t)ys * 4, (cuuint64_t)nx * ys * 4};
    const cuuint32_t b[3] = {(cuuint32_t)box_cols, (cuuint32_t)box_bins, 1};
    const cuuint32_t one[3] = {1, 1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, (void *)base, d, st, b, one,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
               CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Swizzle of boxes whose rows are kc (32 or 64) bf16 channels.
static CUtensorMapSwizzle swizzle_for(int kc) {
    return kc == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
}

// NHWC bf16 tensor [N][H][W][C]: box = kc (32 or 64) channels x box_w x box_h
// pixels of one image, 64 or 128-byte swizzle; false if the CUDA driver refuses it.
bool encode_nhwc_map(CUtensorMap *m, const void *base, int N, int H, int W, int C, int box_w,
                     int box_h, int kc) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc) return false;
    const cuuint64_t d[4] = {(cuuint64_t)C, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)N};
    const cuuint64_t s[3] = {(cuuint64_t)C * 2, (cuuint64_t)W * C * 2, (cuuint64_t)H * W * C * 2};
    const cuuint32_t b[4] = {(cuuint32_t)kc, (cuuint32_t)box_w, (cuuint32_t)box_h, 1};
    const cuuint32_t one[4] = {1, 1, 1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, (void *)base, d, s, b, one,
               CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for(kc),
               CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Tensor maps of one convolution; false if the CUDA driver refuses them (the
// caller then uses the gather kernel).
struct ConvMaps {
    CUtensorMap x, w, y;
};
static bool conv_tensor_maps(const __nv_bfloat16 *x, const __nv_bfloat16 *w, __nv_bfloat16 *y, int N,
                             int H, int Wd, int Cin, int Cout, int ystride, int box_w, int box_h, int kc,
                             ConvMaps *m) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc) return false;
    if (!encode_nhwc_map(&m->x, x, N, H, Wd, Cin, box_w, box_h, kc)) return false;
    const cuuint32_t one[4] = {1, 1, 1, 1};
    const cuuint64_t wd[3] = {(cuuint64_t)Cin, 9, (cuuint64_t)Cout};
    const cuuint64_t ws[2] = {(cuuint64_t)Cin * 2, (cuuint64_t)9 * Cin * 2};
    const cuuint32_t wb[3] = {(cuuint32_t)kc, 1, (cuuint32_t)Cout};
    if (enc(&m->w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, (void *)w, wd, ws, wb, one,
            CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for(kc), CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return false;
    // stores: a warp's 32 pixels x 32 channels
    const cuuint64_t yd[4] = {(cuuint64_t)Cout, (cuuint64_t)Wd, (cuuint64_t)H, (cuuint64_t)N};
    const cuuint64_t row = (cuuint64_t)ystride * 2;
    const cuuint64_t ys[3] = {row, row * Wd, row * Wd * H};
    const cuuint32_t bw = box_w < 32 ? (cuuint32_t)box_w : 32;
    const cuuint32_t yb[4] = {32, bw, 32 / bw, 1};
    return enc(&m->y, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, (void *)y, yd, ys, yb, one,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Width 2^lw of a 128-pixel tile: the widest of those that cover the image with
// the fewest tiles.
static int conv_tile(int H, int Wd) {
    int best = 7;
    long long least = -1;
    for (int lw = 7; lw >= 3; lw--) {
        const int hb = 128 >> lw;
        const long long t = (long long)((Wd + (1 << lw) - 1) >> lw) * ((H + hb - 1) / hb);
        if (least < 0 || t < least) best = lw, least = t;
    }
    return best;
}

static int sm_count() {
    int dev = 0, sms = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

// -1: no tensor maps.
template <int COUT, int R, bool BAND, int KC, int ST>
static int launch_conv_pipe(const __nv_bfloat16 *x, const __nv_bfloat16 *w, const float *bias,
                            __nv_bfloat16 *y, int N, int H, int Wd, int Cin, int lw, int relu,
                            int ystride, int *err, cudaStream_t st) {
    using Cfg = PipeCfg<COUT, R, BAND, KC, ST>;
    const int hb = BAND ? R : (128 >> lw) * R;
    ConvMaps m;
    if (!conv_tensor_maps(x, w, y, N, H, Wd, Cin, COUT, ystride, 1 << lw, BAND ? R + 2 : hb, KC,
                          &m))
        return -1;
    if (int rc = set_smem((const void *)conv3x3_pipe_kernel<COUT, R, BAND, KC, ST>, Cfg::SMEM)) return rc;
    const int wt = (Wd + (1 << lw) - 1) >> lw, ht = (H + hb - 1) / hb, ntiles = N * wt * ht;
    const int sms = sm_count();
    conv3x3_pipe_kernel<COUT, R, BAND, KC, ST><<<ntiles < sms ? ntiles : sms, kPipeThreads, Cfg::SMEM, st>>>(
        m.x, m.w, m.y, bias, H, Wd, Cin, lw, relu, wt, ht, ntiles, err);
    ARECGB_CUDA(cudaGetLastError());
    return 0;
}

// layout: 0 = TMA path; 1 = the gather kernel with (LBO 256, SBO 128) (for
//         validating the descriptor fields); 2 = the gather kernel with
//         (LBO 128, SBO 256) [K-halves 128 B apart, row groups 256 B apart].
int conv3x3_bf16(const void *X, const void *Wt, const float *bias, void *Y, int N, int H, int Wd,
                 int Cin, int Cout, int relu, int layout, int *err, cudaStream_t st, int ystride) {
    if (ystride <= 0) ystride = Cout;
    if (Cin % kConvKC || Cin < kConvKC || N < 1 || H < 1 || Wd < 1 || ystride < Cout ||
        ystride % 8) {
        set_error("conv3x3: Cin must be a positive multiple of 32");
        return ARECGB_ERR_ARG;
    }
    const auto *x = reinterpret_cast<const __nv_bfloat16 *>(X);
    const auto *w = reinterpret_cast<const __nv_bfloat16 *>(Wt);
    auto *y = reinterpret_cast<__nv_bfloat16 *>(Y);
    const int P = N * H * Wd;
    if (layout == 0) {
        int rc = -1;
#define ARECGB_CONV_PIPE(C, R, BAND, KC, ST, LW) \
    rc = launch_conv_pipe<C, R, BAND, KC, ST>(x, w, bias, y, N, H, Wd, Cin, LW, relu, ystride, err, st)
        const int lw = conv_tile(H, Wd);
        const bool wide = Cin % 64 == 0;
        // Bands need widths of 128.  They would run at any height; taking them at multiples
        // of 4 and 2 keeps the order of every size's products, and so its last places.
        // Two tiles share a chunk's weights (48 KB loaded for them instead of 64 at
        // 128 channels) where that leaves every SM a pair.  Bands: as many rows as
        // two stages of their chunks leave room for.
        const bool pairs = (P + 255) / 256 >= sm_count();
        if (Cout == 32 && Wd % 128 == 0 && H % 4 == 0) {
            if (wide) ARECGB_CONV_PIPE(32, 4, true, 64, 2, 7);
            else ARECGB_CONV_PIPE(32, 4, true, 32, 3, 7);
        } else if (Cout == 64 && Wd % 128 == 0 && H % 2 == 0) {
            if (wide) ARECGB_CONV_PIPE(64, 3, true, 64, 2, 7);
            else ARECGB_CONV_PIPE(64, 4, true, 32, 3, 7);
        } else if (Cout == 32) {
            if (wide) ARECGB_CONV_PIPE(32, 2, false, 64, 5, lw);
            else ARECGB_CONV_PIPE(32, 2, false, 32, 8, lw);
        } else if (Cout == 64) {
            if (wide) ARECGB_CONV_PIPE(64, 2, false, 64, 4, lw);
            else ARECGB_CONV_PIPE(64, 2, false, 32, 8, lw);
        } else if (Cout == 128) {
            if (wide && pairs) ARECGB_CONV_PIPE(128, 2, false, 64, 4, lw);
            else if (wide) ARECGB_CONV_PIPE(128, 1, false, 64, 6, lw);
            else ARECGB_CONV_PIPE(128, 2, false, 32, 8, lw);
        } else if (Cout == 256) {
            if (wide) ARECGB_CONV_PIPE(256, 1, false, 64, 4, lw);
            else ARECGB_CONV_PIPE(256, 1, false, 32, 8, lw);
        }
#undef ARECGB_CONV_PIPE
        if (rc >= 0) return rc;
    }
    if (layout == 2) layout = 0;
#define ARECGB_CONV(C)                                                                     \
    if (Cout == C)                                                                         \
        return layout ? launch_conv<C, 256, 128>(x, w, bias, y, H, Wd, Cin, P, relu, ystride, err, st) \
                      : launch_conv<C, 128, 256>(x, w, bias, y, H, Wd, Cin, P, relu, ystride, err, st);
    ARECGB_CONV(32) ARECGB_CONV(64) ARECGB_CONV(128) ARECGB_CONV(256)
#undef ARECGB_CONV
    set_error("conv3x3: Cout must be 32, 64, 128 or 256");
    return ARECGB_ERR_ARG;
}

}  // namespace arecgb

extern "C" int arecgb_conv3x3_bf16(const void *X, const void *Wt, const float *bias, void *Y, int N,
                                   int H, int W, int Cin, int Cout, int relu, int layout, int *err,
                                   void *stream) {
    return arecgb::conv3x3_bf16(X, Wt, bias, Y, N, H, W, Cin, Cout, relu, layout, err,
                                (cudaStream_t)stream, Cout);
}
