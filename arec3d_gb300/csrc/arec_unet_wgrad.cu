// Weight gradient of a 3x3 convolution on the tensor cores:
//
//   gw[co][dy][dx][ci] += sum_p dpre[p][co] * x[p + (dy, dx)][ci]
//
// (x, dpre: NHWC bf16; gw FP32), the contraction over the pixels p, with both
// operands channels-contiguous: tcgen05.mma with MN-major A and B.  M runs over
// (dx, ci) of one dy in tiles of 128, N over co, K over pixels.
//
// A block takes a range of 8x8-pixel chunks (K = 64).  Per chunk, TMA brings for
// each dx the 8 (+ 2) rows of x the block's dy need, in blocks of 64 (or 32)
// channels (pixels outside the image arrive as zeros: the convolution's padding),
// and dpre's blocks (zero outside: ragged chunks add nothing), 128 or 64-byte
// swizzle.  Eight pixels of a block are one swizzle atom, so dy is an offset of
// one atom and a K step of 16 pixels one of two; the blocks of a tile lie one
// region apart.  One thread issues the loads, one warp the MMAs (four K steps per
// chunk and tile, starting from zero); twelve warps add each chunk's accumulators
// from TMEM to FP32 registers (up to 12 blocks of 32 columns, 4 per warp) and at
// the end to gw (FP32 atomics).
//
// The sum over the chunks leaves TMEM because the tensor core's FP32
// accumulation rounds toward zero: with all 431 K steps of a 32 -> 32 layer at
// 16 x 256^2 pixels summed in TMEM the result was 1.4e-5 off FP64 on data of one
// sign (the CUDA-core kernel it replaces 2.0e-7, and 6.0e-7 on data of both
// signs); four steps per chunk and rounded adds give 1.9e-7 and 2.9e-7.
//
// What bounds it: the issue of the MMAs, 45 to 60 clocks each, and two waits of
// about 150 per tile and chunk (1700 clocks per chunk of a 32 -> 32 layer).  Time
// of that layer 3.08 -> 0.09 ms, 256 -> 256 at 16 x 32^2 2.49 -> 0.03 ms, all
// layers of a training batch (16 x 256^2) 58.9 -> 1.16 ms; 1.50 with tile counts
// known at run time only, one hand-over per chunk and 32-channel loads.  Splits:
// dy, ci and co are divided over blocks when their tiles exceed 384 TMEM columns;
// the pixel chunks over as many blocks as fill the SMs.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>

#include "arec_internal.cuh"
#include "arec_umma.cuh"
#include "arec_unet.cuh"

namespace arecgb {

bool encode_nhwc_map(CUtensorMap *m, const void *base, int N, int H, int W, int C, int box_w,
                     int box_h, int kc);

namespace unet {

namespace {

constexpr int kPix = 8;                        // chunk: kPix x kPix pixels
constexpr int kSmemStages = 200 * 1024;
constexpr int kSlack = 16 * 1024;              // unused M blocks of a tile read past the last stage
constexpr uint32_t kWgWait = 4u << 20;

constexpr int kEpiWarps = 12;                  // three warpgroups
constexpr int kBlocks = 12;                    // 32-column accumulator blocks per block at most
constexpr int kWgThreads = 32 * (kEpiWarps + 4);
// the launch's 512 x 128 registers: 12 warps x 32 x 152 + 4 x 32 x 56
constexpr int kRegsEpi = 152, kRegsLow = 56;

// One operand in shared memory: blocks of kc (32 or 64) channels of the chunk's
// pixels, as TMA writes them with the 64 or 128-byte swizzle (MN-major: 8 pixels
// of a block are one swizzle atom).
struct Operand {
    int kc;          // channels of a block
    int row;         // bytes of 8 pixels
    int block;       // bytes of a block
    uint64_t desc;   // descriptor without the address
};

struct WgradJob {
    Operand x, d;
    int cib, cob;        // 32-channel blocks of x and dpre per block
    int ci_jobs, co_jobs;
    int stage, stages;
    int chunks, wt, ht;  // pixel chunks in all, per row, per column
    int bufs;            // accumulator sets in TMEM (2 when they fit)
    uint32_t cols;       // TMEM columns allocated
};

// NDY taps dy (3 or 1) and TILES M tiles (of 128) per dy.  A block's accumulators
// are NDY * TILES tiles of 32 cob columns, handed to the epilogue and back one by
// one: the sums of a tile leave TMEM while the next tile's MMAs run.
template <int NDY, int TILES>
__global__ void __launch_bounds__(kWgThreads, 1)
    k_wgrad_mma(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmD,
                float *__restrict__ gw, int Cin, const WgradJob J, int *err) {
    constexpr int NT = NDY * TILES;
    extern __shared__ unsigned char sm_raw[];
    __shared__ __align__(8) uint64_t full[4], empty[4], accfull[2][NT], accfree[2][NT];
    __shared__ uint32_t tmem_base;
    const uint32_t raw = umma::smem_addr(sm_raw);
    unsigned char *sm = sm_raw + ((1024u - (raw & 1023u)) & 1023u);
    const int tid = threadIdx.x, warp = umma::uniform(tid >> 5), lane = tid & 31;
    int job = blockIdx.y;
    const int dy0 = NDY == 3 ? 0 : job % 3;
    if (NDY != 3) job /= 3;
    const int ci0 = job % J.ci_jobs * J.cib * 32, co0 = job / J.ci_jobs * J.cob * 32;
    const int c_lo = (int)((long long)J.chunks * blockIdx.x / gridDim.x);
    const int nc = (int)((long long)J.chunks * (blockIdx.x + 1) / gridDim.x) - c_lo;
    if (nc < 1) return;  // uniform over the block

    if (warp == 0) {
        umma::tmem_alloc(&tmem_base, J.cols);
        umma::tmem_relinquish();
    }
    if (tid == 0) {
        for (int s = 0; s < J.stages; s++) {
            umma::mbar_init(&full[s], 1);
            umma::mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; b++)
            for (int t = 0; t < NT; t++) {
                umma::mbar_init(&accfull[b][t], 1);
                umma::mbar_init(&accfree[b][t], 4 * J.cob);
            }
        umma::mbar_fence_init();
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = umma::uniform(tmem_base);
    const int N = J.cob * 32, nreg = 3 * J.cib;
    const int nxb = J.cib * 32 / J.x.kc, ndb = J.cob * 32 / J.d.kc;  // blocks per dx, of dpre

    if (warp >= kEpiWarps) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(kRegsLow));
        if (warp == kEpiWarps && lane == 0) {
            for (int it = 0; it < nc; it++) {
                const int c = c_lo + it, s = it % J.stages;
                if (it >= J.stages &&
                    !umma::mbar_wait(&empty[s], (uint32_t)(it / J.stages - 1) & 1u, kWgWait)) {
                    atomicOr(err, 4);
                    umma::ring_drain(full, J.stages, it, kWgWait);
                    break;
                }
                const int w0 = c % J.wt * kPix, h0 = c / J.wt % J.ht * kPix, n = c / (J.wt * J.ht);
                unsigned char *X = sm + (size_t)s * J.stage, *D = X + 3 * nxb * J.x.block;
                umma::mbar_arrive_expect_tx(&full[s], (uint32_t)J.stage);
                for (int dx = 0; dx < 3; dx++)
                    for (int b = 0; b < nxb; b++, X += J.x.block)
                        umma::tma_load_4d(X, &tmX, ci0 + J.x.kc * b, w0 + dx - 1, h0 + dy0 - 1, n, &full[s]);
                for (int b = 0; b < ndb; b++, D += J.d.block)
                    umma::tma_load_4d(D, &tmD, co0 + J.d.kc * b, w0, h0, n, &full[s]);
            }
        } else if (warp == kEpiWarps + 1) {
            // BF16 operands, both MN-major (bits 15, 16)
            const uint32_t idesc = umma::idesc_bf16(128, N) | (1u << 15) | (1u << 16);
            const uint32_t base = umma::uniform(umma::smem_addr(sm));
            // a tile is four 32-channel blocks; a K step two rows of 8 pixels; addresses / 16
            const uint32_t tile = (uint32_t)(128 / J.x.kc * J.x.block) >> 4;
            const uint32_t xrow = (uint32_t)J.x.row >> 4, drow = (uint32_t)J.d.row >> 4;
            bool ok = true;
            for (int it = 0; it < nc && ok; it++) {
                const int s = it % J.stages, b = it % J.bufs, use = it / J.bufs;
                ok = umma::mbar_wait_warp(&full[s], (uint32_t)(it / J.stages) & 1u, kWgWait);
                const uint32_t x = base + (uint32_t)(s * J.stage), d = x + (uint32_t)(3 * nxb * J.x.block);
                const uint64_t xd = J.x.desc | (uint64_t)(x >> 4), dd = J.d.desc | (uint64_t)(d >> 4);
#pragma unroll
                for (int t = 0; t < NT; t++) {
                    if (use > 0)
                        ok = ok && umma::mbar_wait_warp(&accfree[b][t], (uint32_t)(use - 1) & 1u, kWgWait);
                    if (!ok) break;
                    umma::fence_after_sync();
                    const uint64_t a = xd + (uint64_t)(t % TILES * tile + t / TILES * xrow);
                    const uint32_t acc = tmem + (uint32_t)((b * NT + t) * N);
#pragma unroll
                    for (int k = 0; k < kPix / 2; k++)
                        umma::mma_f16_warp(acc, a + (uint64_t)(2 * k * xrow), dd + (uint64_t)(2 * k * drow),
                                           idesc, k > 0 ? 1u : 0u);
                    if (t == NT - 1) umma::mma_commit_warp(&empty[s]);
                    umma::mma_commit_warp(&accfull[b][t]);
                }
            }
            // (the epilogue waits for every tile's MMAs, each of which is committed)
            if (!ok && lane == 0) atomicOr(err, 4);
        }
        __syncwarp();
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(kRegsEpi));
        // warp = 4 * group + w: TMEM lanes 32 w.. are M block 4q + w of a tile
        // (32 input channels of one tap); group g takes accumulator blocks g + 3 i
        const int w = warp & 3, g = warp >> 2, nblk = NT * J.cob;
        const uint32_t base = tmem + ((uint32_t)(32 * w) << 16);
        float acc[kBlocks / 3][32];
#pragma unroll
        for (int i = 0; i < kBlocks / 3; i++)
#pragma unroll
            for (int j = 0; j < 32; j++) acc[i][j] = 0.f;
        bool ok = true;
        for (int it = 0; it < nc && ok; it++) {
            const int b = it % J.bufs;
            const uint32_t ph = (uint32_t)(it / J.bufs) & 1u;
#pragma unroll
            for (int i = 0; i < kBlocks / 3; i++)
                if (g + 3 * i < nblk) {
                    const int t = (g + 3 * i) / J.cob;
                    ok = ok && __all_sync(0xffffffffu, umma::mbar_wait(&accfull[b][t], ph, kWgWait));
                    if (!ok) break;
                    umma::fence_after_sync();
                    const uint32_t col = base + (uint32_t)((b * nblk + g + 3 * i) * 32);
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        float v[16];
                        umma::tmem_ld16(col + 16 * h, v);
#pragma unroll
                        for (int j = 0; j < 16; j++) acc[i][16 * h + j] += v[j];
                    }
                    umma::fence_before_sync();
                    __syncwarp();
                    if (lane == 0) umma::mbar_arrive(&accfree[b][t]);
                }
        }
        if (!ok && lane == 0) atomicOr(err, 4);
        if (ok) {
#pragma unroll
            for (int i = 0; i < kBlocks / 3; i++)
                if (g + 3 * i < nblk) {
                    const int t = (g + 3 * i) / J.cob, cc = (g + 3 * i) % J.cob;
                    const int dy = dy0 + t / TILES, blk = t % TILES * 4 + w;
                    const int tap = dy * 3 + blk / J.cib, ci = ci0 + blk % J.cib * 32 + lane;
                    if (blk < nreg) {
#pragma unroll
                        for (int j = 0; j < 32; j++)
                            atomicAdd(&gw[((size_t)(co0 + cc * 32 + j) * 9 + tap) * Cin + ci],
                                      acc[i][j]);
                    }
                }
        }
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) umma::tmem_dealloc(tmem, J.cols);
}

// An operand of `rows` pixel rows whose channels come in pieces of 32 * blocks: the
// blocks are 64 channels where they can be (TMA takes about two clocks for a row of
// 64 bytes as for one of 128).
Operand make_operand(int blocks, int rows) {
    Operand o;
    o.kc = blocks % 2 ? 32 : 64;
    o.row = kPix * o.kc * 2;
    o.block = rows * o.row;
    // descriptor fields / 16: 64-byte swizzle: blocks along M or N in bits 16.., groups
    // of 8 pixels in bits 32..; 128-byte swizzle the same; version; swizzle
    o.desc = (uint64_t)(o.block >> 4) << 16 | (uint64_t)(o.row >> 4) << 32 | (uint64_t)1 << 46 |
             (uint64_t)(o.kc == 64 ? 2 : 4) << 61;
    return o;
}

template <int NDY, int TILES>
int launch_wgrad(const CUtensorMap &tx, const CUtensorMap &td, float *gw, int Cin, const WgradJob &J,
                 int *err, cudaStream_t st) {
    if (int rc = set_smem((const void *)k_wgrad_mma<NDY, TILES>, kSmemStages + kSlack + 1024)) return rc;
    const int jobs = J.ci_jobs * J.co_jobs * (3 / NDY);
    const int splits = std::max(1, std::min(J.chunks, 152 / jobs));
    k_wgrad_mma<NDY, TILES><<<dim3(splits, jobs), kWgThreads, J.stages * J.stage + kSlack + 1024, st>>>(
        tx, td, gw, Cin, J, err);
    ARECGB_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace

int conv_wgrad(const __nv_bfloat16 *x, const __nv_bfloat16 *dpre, float *gw, int N, int H, int W,
               int Cin, int Cout, int *err, cudaStream_t st) {
    WgradJob J;
    J.cib = std::min(4, Cin / 32);
    J.cob = std::min(4, Cout / 32);
    J.ci_jobs = Cin / (32 * J.cib);
    J.co_jobs = Cout / (32 * J.cob);
    const int tiles = (3 * J.cib + 3) / 4, ndy = 3 * tiles * J.cob <= kBlocks ? 3 : 1;
    J.x = make_operand(J.cib, kPix + ndy - 1);
    J.d = make_operand(J.cob, kPix);
    J.stage = 3 * J.cib * 32 / J.x.kc * J.x.block + J.cob * 32 / J.d.kc * J.d.block;
    J.stages = std::min(4, kSmemStages / J.stage);
    J.wt = (W + kPix - 1) / kPix;
    J.ht = (H + kPix - 1) / kPix;
    J.chunks = N * J.wt * J.ht;
    const int set = ndy * tiles * J.cob * 32;  // columns of one accumulator set, <= 384
    J.bufs = 2 * set <= 512 ? 2 : 1;
    J.cols = 32;
    while (J.cols < (uint32_t)(J.bufs * set)) J.cols *= 2;
    CUtensorMap tx, td;
    if (!encode_nhwc_map(&tx, x, N, H, W, Cin, kPix, kPix + ndy - 1, J.x.kc) ||
        !encode_nhwc_map(&td, dpre, N, H, W, Cout, kPix, kPix, J.d.kc)) {
        set_error("conv_wgrad: tensor map encoding failed");
        return ARECGB_ERR_ARG;
    }
#define ARECGB_WGRAD(D, T) \
    if (ndy == D && tiles == T) return launch_wgrad<D, T>(tx, td, gw, Cin, J, err, st);
    ARECGB_WGRAD(3, 1) ARECGB_WGRAD(3, 2) ARECGB_WGRAD(3, 3) ARECGB_WGRAD(1, 2) ARECGB_WGRAD(1, 3)
#undef ARECGB_WGRAD
    set_error("conv_wgrad: unsupported channel counts");
    return ARECGB_ERR_ARG;
}

}  // namespace unet
}  // namespace arecgb
