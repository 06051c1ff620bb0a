// Weight gradient of a 3x3 convolution on the tensor cores:
//
//   gw[co][dy][dx][ci] += sum_p dpre[p][co] * x[p + (dy, dx)][ci]
//
// (x, dpre: NHWC bf16; gw FP32), the contraction over the pixels p, with both
// operands channels-contiguous: tcgen05.mma with MN-major A and B.  M runs over
// (dx, ci) of one dy in tiles of 128, N over co, K over pixels.
//
// A block takes a range of 8x8-pixel chunks (K = 64).  Per chunk, TMA brings
// for each dx and 32-channel block of x the 8 (+ 2) rows the block's dy need
// (pixels outside the image arrive as zeros: the convolution's padding), and
// dpre's blocks (zero outside: ragged chunks add nothing), 64-byte swizzle.
// Eight pixels of a 32-channel block are one 512-byte swizzle atom, so dy is an
// offset of 512 bytes and a K step of 16 pixels one of 1024; the 32-channel
// blocks of a tile lie one region apart.  One thread issues the loads, one warp the
// MMAs (four K steps per chunk and tile, starting from zero); twelve warps add
// each chunk's accumulators from TMEM to FP32 registers (up to 12 blocks of 32
// columns, 4 per warp) and at the end to gw (FP32 atomics).
//
// The sum over the chunks leaves TMEM because the tensor core's FP32
// accumulation rounds toward zero: with all 431 K steps of a 32 -> 32 layer at
// 16 x 256^2 pixels summed in TMEM the result was 1.4e-5 off FP64 on data of one
// sign (the CUDA-core kernel it replaces 2.0e-7, and 6.0e-7 on data of both
// signs); four steps per chunk and rounded adds give 1.9e-7 and 2.9e-7.
// Time of that layer 3.08 -> 0.21 ms, 256 -> 256 at 16 x 32^2 2.49 -> 0.08 ms,
// one training batch's gradient (16 x 256^2) 63.5 -> 6.5 ms; with the MMAs issued by
// a whole warp all layers of it take 1.50 ms instead of 1.90.  Splits: dy, ci and co
// are divided over blocks when their tiles exceed 384 TMEM columns; the pixel chunks
// over as many blocks as fill the SMs.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <mutex>

#include "arec_internal.cuh"
#include "arec_umma.cuh"
#include "arec_unet.cuh"

namespace arecgb {

bool encode_nhwc_map(CUtensorMap *m, const void *base, int N, int H, int W, int C, int box_w,
                     int box_h, int kc);

namespace unet {

namespace {

constexpr int kPix = 8;                        // chunk: kPix x kPix pixels
constexpr int kAtom = kPix * 64;               // one row of a chunk: 8 pixels x 32 channels
constexpr int kDBlock = kPix * kAtom;          // dpre: 64 pixels x 32 channels
constexpr int kSmemStages = 200 * 1024;
constexpr int kSlack = 16 * 1024;              // unused M blocks of a tile read past the last stage
constexpr uint32_t kWgWait = 4u << 20;

constexpr int kEpiWarps = 12;                  // three warpgroups
constexpr int kBlocks = 12;                    // 32-column accumulator blocks per block at most
constexpr int kWgThreads = 32 * (kEpiWarps + 2);

struct WgradJob {
    int cib, cob;        // 32-channel blocks of x and dpre per block
    int ndy;             // taps dy per block (3 or 1)
    int tiles;           // M tiles (of 128) per dy: ceil(3 cib / 4)
    int ci_jobs, co_jobs;
    int region, stage, stages;
    int chunks, wt, ht;  // pixel chunks in all, per row, per column
    int bufs;            // accumulator sets in TMEM (2 when they fit)
    uint32_t cols;       // TMEM columns allocated
};

// K-major is the descriptor of arec_umma.cuh; here the operand is MN-major:
// 32-channel (64-byte) blocks `lbo` bytes apart, groups of 8 pixels 512 bytes.
__device__ __forceinline__ uint64_t desc_mn_sw64(uint32_t saddr, uint32_t lbo) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFF);
    d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)(512 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;
    return d;
}

__global__ void __launch_bounds__(kWgThreads, 1)
    k_wgrad_mma(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmD,
                float *__restrict__ gw, int Cin, WgradJob J, int *err) {
    extern __shared__ unsigned char sm_raw[];
    __shared__ __align__(8) uint64_t full[4], empty[4], accfull[2], accfree[2];
    __shared__ uint32_t tmem_base;
    const uint32_t raw = umma::smem_addr(sm_raw);
    unsigned char *sm = sm_raw + ((1024u - (raw & 1023u)) & 1023u);
    const int tid = threadIdx.x, warp = umma::uniform(tid >> 5), lane = tid & 31;
    int job = blockIdx.y;
    const int dy0 = J.ndy == 3 ? 0 : job % 3;
    if (J.ndy != 3) job /= 3;
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
        for (int b = 0; b < 2; b++) {
            umma::mbar_init(&accfull[b], 1);
            umma::mbar_init(&accfree[b], kEpiWarps);
        }
        umma::mbar_fence_init();
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = tmem_base;
    const int N = J.cob * 32, nreg = 3 * J.cib;
    const int nblk = J.ndy * J.tiles * J.cob;  // accumulator blocks (32 columns each)

    if (warp == kEpiWarps) {
        if (lane == 0)
            for (int it = 0; it < nc; it++) {
                const int c = c_lo + it, s = it % J.stages;
                if (it >= J.stages &&
                    !umma::mbar_wait(&empty[s], (uint32_t)(it / J.stages - 1) & 1u, kWgWait)) {
                    atomicOr(err, 4);
                    break;
                }
                const int w0 = c % J.wt * kPix, h0 = c / J.wt % J.ht * kPix, n = c / (J.wt * J.ht);
                unsigned char *X = sm + (size_t)s * J.stage, *D = X + nreg * J.region;
                umma::mbar_arrive_expect_tx(&full[s], (uint32_t)J.stage);
                for (int dx = 0; dx < 3; dx++)
                    for (int b = 0; b < J.cib; b++)
                        umma::tma_load_4d(X + (dx * J.cib + b) * J.region, &tmX, ci0 + 32 * b,
                                          w0 + dx - 1, h0 + dy0 - 1, n, &full[s]);
                for (int b = 0; b < J.cob; b++)
                    umma::tma_load_4d(D + b * kDBlock, &tmD, co0 + 32 * b, w0, h0, n, &full[s]);
            }
        __syncwarp();
    } else if (warp == kEpiWarps + 1) {
        // BF16 operands, both MN-major (bits 15, 16)
        const uint32_t idesc = umma::idesc_bf16(128, N) | (1u << 15) | (1u << 16);
        const uint32_t tm = umma::uniform(tmem), base = umma::uniform(umma::smem_addr(sm));
        for (int it = 0; it < nc; it++) {
            const int s = it % J.stages, b = it % J.bufs, use = it / J.bufs;
            if (!umma::mbar_wait_warp(&full[s], (uint32_t)(it / J.stages) & 1u, kWgWait) ||
                (use > 0 && !umma::mbar_wait_warp(&accfree[b], (uint32_t)(use - 1) & 1u, kWgWait))) {
                if (lane == 0) atomicOr(err, 4);
                break;
            }
            umma::fence_after_sync();
            const uint32_t x = base + (uint32_t)(s * J.stage), d = x + nreg * J.region;
#pragma unroll
            for (int k = 0; k < kPix * kPix / 16; k++) {
                const uint64_t bd = desc_mn_sw64(d + k * 1024, kDBlock);
                for (int dy = 0; dy < J.ndy; dy++)
                    for (int q = 0; q < J.tiles; q++)
                        umma::mma_f16_warp(
                            tm + (uint32_t)(b * nblk * 32 + (dy * J.tiles + q) * N),
                            desc_mn_sw64(x + 4 * q * J.region + dy * kAtom + k * 1024, J.region), bd,
                            idesc, k > 0 ? 1u : 0u);
            }
            umma::mma_commit_warp(&empty[s]);
            umma::mma_commit_warp(&accfull[b]);
        }
        __syncwarp();
    } else {
        // warp = 4 * group + w: TMEM lanes 32 w.. are M block 4q + w of a tile
        // (32 input channels of one tap); group g takes accumulator blocks g + 3 i
        const int w = warp & 3, g = warp >> 2;
        const uint32_t base = tmem + ((uint32_t)(32 * w) << 16);
        float acc[kBlocks / 3][32];
#pragma unroll
        for (int i = 0; i < kBlocks / 3; i++)
#pragma unroll
            for (int j = 0; j < 32; j++) acc[i][j] = 0.f;
        bool ok = true;
        for (int it = 0; it < nc && ok; it++) {
            const int b = it % J.bufs;
            ok = __all_sync(0xffffffffu,
                            umma::mbar_wait(&accfull[b], (uint32_t)(it / J.bufs) & 1u, kWgWait));
            if (!ok) break;
            umma::fence_after_sync();
#pragma unroll
            for (int i = 0; i < kBlocks / 3; i++)
                if (g + 3 * i < nblk) {
                    const uint32_t col = base + (uint32_t)((b * nblk + g + 3 * i) * 32);
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        float v[16];
                        umma::tmem_ld16(col + 16 * h, v);
#pragma unroll
                        for (int j = 0; j < 16; j++) acc[i][16 * h + j] += v[j];
                    }
                }
            umma::fence_before_sync();
            __syncwarp();
            if (lane == 0) umma::mbar_arrive(&accfree[b]);
        }
        if (!ok && lane == 0) atomicOr(err, 4);
        if (ok) {
#pragma unroll
            for (int i = 0; i < kBlocks / 3; i++)
                if (g + 3 * i < nblk) {
                    const int t = (g + 3 * i) / J.cob, cc = (g + 3 * i) % J.cob;
                    const int dy = dy0 + t / J.tiles, blk = t % J.tiles * 4 + w;
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

}  // namespace

int conv_wgrad(const __nv_bfloat16 *x, const __nv_bfloat16 *dpre, float *gw, int N, int H, int W,
               int Cin, int Cout, int *err, cudaStream_t st) {
    WgradJob J;
    J.cib = std::min(4, Cin / 32);
    J.cob = std::min(4, Cout / 32);
    J.ci_jobs = Cin / (32 * J.cib);
    J.co_jobs = Cout / (32 * J.cob);
    J.tiles = (3 * J.cib + 3) / 4;
    J.ndy = 3 * J.tiles * J.cob <= kBlocks ? 3 : 1;
    J.region = (kPix + J.ndy - 1) * kAtom;
    J.stage = 3 * J.cib * J.region + J.cob * kDBlock;
    J.stages = std::min(4, kSmemStages / J.stage);
    J.wt = (W + kPix - 1) / kPix;
    J.ht = (H + kPix - 1) / kPix;
    J.chunks = N * J.wt * J.ht;
    const int set = J.ndy * J.tiles * J.cob * 32;  // columns of one accumulator set, <= 384
    J.bufs = 2 * set <= 512 ? 2 : 1;
    J.cols = 32;
    while (J.cols < (uint32_t)(J.bufs * set)) J.cols *= 2;
    CUtensorMap tx, td;
    if (!encode_nhwc_map(&tx, x, N, H, W, Cin, kPix, kPix + J.ndy - 1, 32) ||
        !encode_nhwc_map(&td, dpre, N, H, W, Cout, kPix, kPix, 32)) {
        set_error("conv_wgrad: tensor map encoding failed");
        return ARECGB_ERR_ARG;
    }
    const int smem = J.stages * J.stage + kSlack + 1024;
    static std::once_flag once;
    static cudaError_t attr = cudaSuccess;
    std::call_once(once, [] {
        attr = cudaFuncSetAttribute(k_wgrad_mma, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    kSmemStages + kSlack + 1024);
    });
    ARECGB_CUDA(attr);
    const int jobs = J.ci_jobs * J.co_jobs * (3 / J.ndy);
    const int splits = std::max(1, std::min(J.chunks, 152 / jobs));
    k_wgrad_mma<<<dim3(splits, jobs), kWgThreads, smem, st>>>(tx, td, gw, Cin, J, err);
    ARECGB_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace unet
}  // namespace arecgb
