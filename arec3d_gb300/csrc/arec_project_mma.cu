// Projectors on the tensor cores: FP16 split of the operand, forward
// projection (see arec_project_mma.cuh for the idea).
//
// Forward projection  q[a][b][y] += sum_k w(k, a, b) x[k][y].
//   D[y][(a, j)] = sum over the rays k of a block of X[y][k] W[k][(a, j)]:
//   M = 128 slices, N = 16 bins x up to 8 angles, K = 64 rays.
// Angles are taken in groups (one or two of the plan's 4-angle groups); lines
// (rows when |cos| >= |sin|, else columns) in blocks of 8; and the pixels of a
// line block in blocks of 8 whose start follows the group's middle angle from
// line block to line block, so that such a strip of 8 x 8 blocks projects into
// about the same bins all the way.  A segment is a run of line blocks over which
// every angle's footprint stays inside one 16-bin window; its sums are added to
// q at its end.  Strips three apart have disjoint windows in a segment, so a
// launch takes one segment number and every third strip: no two blocks of a
// launch add to the same bins, and launches follow one another in a fixed order
// (results do not depend on timing).
#include <math.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <mutex>
#include <numeric>
#include <vector>

#include "arec_project_mma.cuh"
#include "arec_umma.cuh"
#include "arec_weights.cuh"

#include "arec_project_args.cuh"

namespace arecgb {

bool encode_half_map(CUtensorMap *m, const void *base, int ys, int n1, int n2, int box1, int box2);
bool encode_foot_map(CUtensorMap *m, const void *base, int nx, int groups, int na, int box_bins);
// arec_project_{kb,sq}.cu
int launch_wide_kb(const OpArgs &, int, int, int, int, const float *, float *, bool, const WideArgs &,
                   cudaStream_t);
int launch_wide_sq(const OpArgs &, int, int, int, int, const float *, float *, bool, const WideArgs &,
                   cudaStream_t);

namespace {

constexpr int kWin = 16;       // bins of a window
constexpr int kSpread = 13;    // window slots a block's first bins may take: 0 .. 13
constexpr uint32_t kMmaWait = 1u << 22;
// Warps of a block: 8 take sums, 8 build weights, one loads, one issues MMAs (two
// idle: registers are handed over by groups of four warps).
constexpr int kTakers = 8, kBuilders = 8, kLoadWarp = 16, kMmaWarp = 17;
constexpr int kMmaThreads = 32 * 20;
// The tensor core's rounding toward zero takes part of every sum: at 129 to 512 pixels
// 8.4e-8 to 9.3e-8 of a forward projection of data of one sign (random values, spheres,
// a reconstruction), 7.0e-8 with both signs, 3.8e-8 at 5 % of the rays (back 4.5e-8 to
// 5.3e-8, 4.7e-8, 3.6e-8), nothing of sums that are exact.  The conversion adds this share
// of a value to its low half (where some of it is rounded away again): the same for
// every ray and angle, so A and A^T stay transposes of each other but for their scale,
// and set for data of one sign, whose projections lose or gain 0.5e-8 at most: b - A x0
// of a warm start multiplies that (4 steps of Kaiser-Bessel CGLS from there at 65 bins:
// 3.7e-7 from FP64; 3.2e-6 with factors on some of the sums, 3.0e-5 with none).  Errors
// against FP64 at 256 pixels, 64 angles: dense 6.5e-8 and 4.1e-8 back (1.09e-7 and 6.4e-8
// without, FP32 kernels 1.34e-7 and 1.66e-7), 5 % of the rays 7.5e-8 and 5.3e-8 (7.0e-8,
// 6.3e-8; 4.8e-8, 5.2e-8), single rays 9.4e-8 and 6.4e-8 (5.4e-8, 5.3e-8; 4.3e-8, 4.0e-8):
// what lost nothing is off by the share and its rounding, less than one last place.
constexpr float kLostForward = 9e-8f, kLostBack = 5.5e-8f;
constexpr int kSegBlocks = 64;  // line blocks of a segment at most

// ---------------------------------------------------------------------------
// FP16 pairs.

// A pair keeps its 22 bits down to 2^-29 of the slice's largest magnitude (scaled:
// 2^14 .. 2^15).  A slice more than 1/32 of whose nonzero values lie below kSmall
// (2^-30 of the largest, or a little more) would lose bits that FP32 keeps: a fill
// value or a hot pixel beside ordinary data.  Fewer do not matter: values spread
// around zero reach below it in about 2^-28 of the cases, the rounding noise that an
// FP32 transform leaves on a background of zeros (2^-25 of the largest) in 2 %.
constexpr float kSmall = 1.f / 32768.f;
constexpr int kScoreSmall = 32;
constexpr int kScoreShared = 4096;  // slices whose scores a block adds up in shared memory

// Per plan and direction, beside the operand: zeroed before the largest magnitudes are
// taken; mma_stats_bytes.
struct HalfStats {
    unsigned *maxb;              // [ys] largest magnitude per slice
    unsigned long long *score;   // [ys] see add_score
    int *wide;                   // set when one is positive: the operand takes FP32 kernels
    int ys;
};

// Largest magnitude per slice (as ordered integers; an infinity or NaN is >=
// 0x7f800000) of rows [n][ys]; out zeroed by the caller.
__global__ void __launch_bounds__(256)
    k_slice_max(const float4 *__restrict__ v, size_t n, int ys4, unsigned *__restrict__ out,
                const int *skip) {
    extern __shared__ unsigned sm_max[];
    if (skip && *skip) return;
    const int nv = min(ys4, 256), rb = 256 / nv;
    for (int c0 = 0; c0 < ys4; c0 += nv) {
        const int w = min(nv, ys4 - c0), c = threadIdx.x % nv, r0 = threadIdx.x / nv;
        for (int i = threadIdx.x; i < 4 * nv; i += 256) sm_max[i] = 0u;
        __syncthreads();
        if (r0 < rb && c < w) {
            unsigned m0 = 0, m1 = 0, m2 = 0, m3 = 0;
            for (size_t r = (size_t)blockIdx.x * rb + r0; r < n; r += (size_t)gridDim.x * rb) {
                const float4 x = v[r * ys4 + c0 + c];
                m0 = max(m0, __float_as_uint(fabsf(x.x)));
                m1 = max(m1, __float_as_uint(fabsf(x.y)));
                m2 = max(m2, __float_as_uint(fabsf(x.z)));
                m3 = max(m3, __float_as_uint(fabsf(x.w)));
            }
            atomicMax(&sm_max[4 * c], m0);
            atomicMax(&sm_max[4 * c + 1], m1);
            atomicMax(&sm_max[4 * c + 2], m2);
            atomicMax(&sm_max[4 * c + 3], m3);
        }
        __syncthreads();
        for (int i = threadIdx.x; i < 4 * w; i += 256)
            if (sm_max[i]) atomicMax(&out[4 * c0 + i], sm_max[i]);
        __syncthreads();
    }
}

__device__ __forceinline__ unsigned pack_half(float a, float b, float &ra, float &rb) {
    const __half ha = __float2half_rn(a), hb = __float2half_rn(b);
    ra = a - __half2float(ha);
    rb = b - __half2float(hb);
    return (unsigned)__half_as_ushort(ha) | ((unsigned)__half_as_ushort(hb) << 16);
}

// A slice's score: kScoreSmall for every nonzero value below kSmall, less 1 for every
// nonzero value.  A block adds it up in shared memory (cnt: a counter per slice), or
// straight in S.score when there are too many slices for that.
__device__ __forceinline__ void add_score(const HalfStats &S, int *cnt, int slice, int v) {
    if (S.ys <= kScoreShared) atomicAdd(cnt + slice, v);
    else atomicAdd(S.score + slice, (unsigned long long)(long long)v);
}

// A thread's eight slices 8 m ..: their scales and its nonzero values, two counts of 16
// bits to a register (a thread of a grid as large as those below has less than 2^16
// rows of anything that fits the memory).
struct HalfLane {
    float scale[8];
    unsigned count[4] = {0, 0, 0, 0};
    int m;

    __device__ __forceinline__ HalfLane(const HalfStats &S, int m_) : m(m_) {
#pragma unroll
        for (int i = 0; i < 8; i++) scale[i] = pow2f(half_shift(S.maxb[8 * m + i]));
    }
    // Scaled, high and low halves (with `share` of the value more).
    __device__ __forceinline__ void pair(const float4 *v, float share, const HalfStats &S, int *cnt, uint4 &hi,
                                         uint4 &lo) {
        const float4 a = v[0], b = v[1];
        const float raw[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        float f[8], l[8], d0, d1;
        unsigned small = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            f[i] = raw[i] * scale[i];
            if (raw[i] != 0.f) {
                count[i >> 1] += i & 1 ? 0x10000u : 1u;
                if (fabsf(f[i]) < kSmall) small |= 1u << i;
            }
        }
        hi.x = pack_half(f[0], f[1], l[0], l[1]);
        hi.y = pack_half(f[2], f[3], l[2], l[3]);
        hi.z = pack_half(f[4], f[5], l[4], l[5]);
        hi.w = pack_half(f[6], f[7], l[6], l[7]);
#pragma unroll
        for (int i = 0; i < 8; i++) l[i] = fmaf(f[i], share, l[i]) * kLowScale;
        lo.x = pack_half(l[0], l[1], d0, d1);
        lo.y = pack_half(l[2], l[3], d0, d1);
        lo.z = pack_half(l[4], l[5], d0, d1);
        lo.w = pack_half(l[6], l[7], d0, d1);
        for (; small; small &= small - 1) add_score(S, cnt, 8 * m + __ffs(small) - 1, kScoreSmall);
    }
    __device__ __forceinline__ void finish(const HalfStats &S, int *cnt) const {
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int n = (int)(count[i >> 1] >> (i & 1 ? 16 : 0) & 0xffffu);
            if (n) add_score(S, cnt, 8 * m + i, -n);
        }
    }
};

// Before the block's first and after its last values.
__device__ __forceinline__ void start_scores(const HalfStats &S, int *cnt) {
    if (S.ys <= kScoreShared)
        for (int i = threadIdx.x; i < S.ys; i += 256) cnt[i] = 0;
    __syncthreads();
}
__device__ __forceinline__ void finish_scores(const HalfStats &S, const int *cnt) {
    __syncthreads();
    if (S.ys <= kScoreShared)
        for (int i = threadIdx.x; i < S.ys; i += 256)
            if (cnt[i]) atomicAdd(S.score + i, (unsigned long long)(long long)cnt[i]);
    if (blockIdx.x == 0)
        for (int i = threadIdx.x; i < S.ys; i += 256)
            if (S.maxb[i] >= kWideBits) atomicAdd(S.score + i, 1ull << 62);
}

// Rows [n][ys] as FP16 pairs [2][rows][ys], row r at place[r].  The grid's threads are a
// multiple of ys8: each keeps its slices.
__global__ void __launch_bounds__(256)
    k_to_half(const float4 *__restrict__ v, size_t n, int ys8, const HalfStats S,
              const int *__restrict__ place, size_t rows, uint4 *__restrict__ out, const int *skip) {
    extern __shared__ int sm_score[];
    if (skip && *skip) return;
    start_scores(S, sm_score);
    const size_t total = n * ys8, t0 = (size_t)blockIdx.x * 256 + threadIdx.x;
    const int m = (int)(t0 % ys8);
    HalfLane h(S, m);
    for (size_t t = t0; t < total; t += (size_t)gridDim.x * 256) {
        uint4 hi, lo;
        h.pair(v + 2 * t, kLostForward, S, sm_score, hi, lo);
        const size_t o = (size_t)place[t / ys8] * ys8 + m;
        out[o] = hi;
        out[rows * ys8 + o] = lo;
    }
    h.finish(S, sm_score);
    finish_scores(S, sm_score);
}

// The sinogram [na][nx][ys] as FP16 pairs [2][na][ys/8][nx][8] (the back
// projector's windows start at any bin: eight slices of neighbouring bins lie in
// one row).  A warp takes 8 bins x 4 slice groups: 128-byte pieces on both sides.
// The grid's warps are a multiple of the groups of four: each keeps its own.
__global__ void __launch_bounds__(256)
    k_sino_to_half(const float4 *__restrict__ v, int na, int nx, int ys8, const HalfStats S,
                   uint4 *__restrict__ out, const int *skip) {
    extern __shared__ int sm_score[];
    if (skip && *skip) return;
    start_scores(S, sm_score);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nmb = (ys8 + 3) / 4, nbb = (nx + 7) / 8;
    const size_t total = (size_t)na * nbb * nmb, half = (size_t)na * ys8 * nx;
    const size_t t0 = (size_t)blockIdx.x * 8 + warp;
    const int m = (int)(t0 % nmb) * 4 + (lane & 3);
    if (m < ys8) {
        HalfLane h(S, m);
        for (size_t t = t0; t < total; t += (size_t)gridDim.x * 8) {
            const int b = (int)(t / nmb % nbb) * 8 + (lane >> 2);
            const size_t a = t / nmb / nbb;
            if (b >= nx) continue;
            uint4 hi, lo;
            h.pair(v + ((a * nx + b) * ys8 + m) * 2, kLostBack, S, sm_score, hi, lo);
            const size_t o = (a * ys8 + m) * nx + b;
            out[o] = hi;
            out[half + o] = lo;
        }
        h.finish(S, sm_score);
    }
    finish_scores(S, sm_score);
}

// ---------------------------------------------------------------------------
// Forward projection.

// No-swizzle MN-major operand: 8 (M or N) x 8 (K) FP16 cores of 128 bytes, the
// 8 elements of M or N contiguous; `mn` bytes between cores along M or N, `k`
// along K.
__device__ __forceinline__ uint64_t desc_mn(uint32_t saddr, uint32_t mn, uint32_t k) {
    return umma::smem_desc(saddr, k, mn);
}
// MN-major operand with the 128-byte swizzle, as a TMA load of 64-element rows
// writes it: atoms of 64 (M) x 8 (K) elements, 1024 bytes; `mn` bytes between
// atoms along M, `k` along K.  Bases are multiples of 1024.
__device__ __forceinline__ uint64_t desc_mn_sw128(uint32_t saddr, uint32_t mn, uint32_t k) {
    return umma::smem_desc(saddr, mn, k) | (uint64_t)2 << 61;
}
// FP16 operands, FP32 accumulator, both MN-major (bits 15, 16).
__device__ __forceinline__ uint32_t idesc_f16(int N) {
    return (1u << 4) | (1u << 15) | (1u << 16) | ((uint32_t)(N >> 3) << 17) | ((128u >> 4) << 24);
}

// Taps as FP16 pairs: (centre bin, hi w0 | hi w1 << 16, lo w0 | lo w1 << 16,
// hi w2 | lo w2 << 16), weights scaled by kWeightScale.
__device__ __forceinline__ uint4 pack_taps(const Taps &t) {
    float l0, l1, l2, z, d0, d1;
    const unsigned h01 = pack_half(t.w0 * kWeightScale, t.w1 * kWeightScale, l0, l1);
    const unsigned h2 = pack_half(t.w2 * kWeightScale, 0.f, l2, z);
    const unsigned l01 = pack_half(l0 * kLowScale, l1 * kLowScale, d0, d1);
    const unsigned lo2 = pack_half(l2 * kLowScale, 0.f, d0, d1);
    return make_uint4((unsigned)t.iqx, h01, l01, h2 | lo2 << 16);
}

// The plan's taps table: [4-angle group][ray in the group's line order][4].
template <int W>
__global__ void __launch_bounds__(256) k_packed_taps(OpArgs A, uint4 *taps) {
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (size_t)A.ngroups * A.nrays * kGroupAngles) return;
    const int j = (int)(t % kGroupAngles);
    const size_t gk = t / kGroupAngles;
    const int grp = (int)(gk / A.nrays), k = (int)(gk % A.nrays);
    const int4 G = A.groups[grp];
    taps[t] = j < G.y ? pack_taps(ray_taps<W>(A.ray[G.z ? A.kinv[k] : k], A.ang[G.x + j], A.r_hi, A.r_lo))
                      : make_uint4(0u, 0u, 0u, 0u);
}

// The 16-slot rows (hi and, `part` bytes on, lo) of one (ray, angle): packed taps
// e at slots p, p+1, p+2 (p in [0, 13]), each row two cores of 16 bytes at d and
// d + 128.  The weights fill words q = p / 2 and q + 1 of a row's eight: the core
// that holds word q gets them by two conditional moves (q & 1, q & 2), the other
// at most their end.
__device__ __forceinline__ void store_rows(unsigned char *d, int part, int p, const uint4 &e) {
    const bool odd = p & 1, b0 = p & 2, b1 = p & 4;
    unsigned char *da = d + (p >> 3) * 128, *db = d + (1 - (p >> 3)) * 128;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const unsigned ab = h ? e.z : e.y, c = h ? e.w >> 16 : e.w & 0xffffu;
        const unsigned lo = odd ? ab << 16 : ab, hi = odd ? __funnelshift_l(ab, c, 16) : c;
        const unsigned s0 = b0 ? 0u : lo, s1 = b0 ? lo : hi, s2 = b0 ? hi : 0u;
        *reinterpret_cast<uint4 *>(da + h * part) =
            make_uint4(b1 ? 0u : s0, b1 ? 0u : s1, b1 ? s0 : s2, b1 ? s1 : 0u);
        *reinterpret_cast<uint4 *>(db + h * part) = make_uint4(b1 ? s2 : 0u, 0u, 0u, 0u);
    }
}

template <int R>
__device__ __forceinline__ void regs_dec() {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(R));
}
template <int R>
__device__ __forceinline__ void regs_inc() {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(R));
}

// A line of the sweep: first ray of the line in the sweep's ray order and the
// pixels [lo, hi] it holds (rows or columns of the disk).
__device__ __forceinline__ void line_info(const OpArgs &A, int orient, int li, int &start, int &lo,
                                          int &hi) {
    start = 0;
    lo = 1 << 20;
    hi = -1;
    if (li >= A.nx) return;
    if (orient == 0) {
        const RowInfo r = A.rows[li];
        start = r.start; lo = r.lo; hi = r.hi;
    } else {
        const ColInfo c = A.cols[li];
        start = c.start; lo = c.lo; hi = c.hi;
    }
}

template <int MT>
struct FpMma {
    static constexpr int SUB = 16 * 1024;            // 64 pixels x 128 slices, one part
    static constexpr int NSUB = 2 * MT;              // (M tile, part: lo first)
    static constexpr int X = NSUB * SUB;
    static constexpr int B = 32 * 1024;              // [part][8 rows][16 N-cores][128 B]
    static constexpr int STAGE = X + B;
    static constexpr int STAGES = MT == 2 ? 2 : 3;
    static constexpr int SMEM = STAGES * STAGE + 1024;
    static constexpr uint32_t COLS = MT * 256;       // two accumulator sets of MT x 128 columns
    static constexpr int ACC = MT * 64;              // accumulators per taker thread
    // launched with 96 registers x 640 threads = 61440; 12 warps x 32 x 56 + 8 x 32 x 152 = 60416
    static constexpr int REGS_LOW = 56, REGS_TAKE = 152;
};

// Block: one group, strip and segment x MT * 128 slices.  One thread loads (per M
// tile and part two TMA boxes of 8 x 8 pixels x 64 slices from the FP16 image
// stack; a block's K index is its row-major pixel whatever the sweep), one issues
// the MMAs, the builders write the weights of the next block (warp = its row,
// lane = column and angle, two angles each) and the takers add a block's sums to
// registers (thread = slice, columns = (angle, bin)).
//
// What bounds it: the shared memory's 128 bytes per clock.  Per block of rays,
// 8 angles and 256 slices the MMAs read 24 x 8 KB and the loads and builders
// write 64 + 32 KB: 2300 clocks, against 1536 of tensor work (measured: 3000, and
// a segment's end, adds to q, about a fifth of the whole).  A projection at
// 1024^2 x 1200 angles x 512 slices takes 43.8 ms, 159.6 with the FP32 kernels,
// which the FMA pipes bound.
template <int W, int MT>
__global__ void __launch_bounds__(kMmaThreads, 1)
    fp_mma_kernel(OpArgs A, MmaPlan M, const __grid_constant__ CUtensorMap tmx, float *__restrict__ q,
                  const unsigned *__restrict__ maxb, const int *__restrict__ wide, int seg,
                  int color) {
    using C = FpMma<MT>;
    extern __shared__ unsigned char sm_raw[];
    __shared__ __align__(8) uint64_t xfull[C::STAGES][C::NSUB], xempty[C::STAGES][C::NSUB];
    __shared__ __align__(8) uint64_t bfull[C::STAGES], bempty[C::STAGES], accfull[2], accfree[2], drained;
    __shared__ uint32_t tmem_base;
    // per line block of the segment and line: ray of the strip's first pixel
    // (of pixel p: that plus p), and the pixels that are rays, first | last << 8
    __shared__ int s_ray[kSegBlocks][8];
    __shared__ unsigned short s_px[kSegBlocks][8];
    __shared__ short blist[kSegBlocks];
    __shared__ unsigned s_any[2];
    __shared__ int s_base[8];
    const int tid = threadIdx.x, warp = umma::uniform(tid >> 5), lane = tid & 31;
    const int g = blockIdx.x % M.ngroups, strip = blockIdx.x / M.ngroups * 3 + color;
    const int4 G = M.groups[g];
    const int2 js = M.strips[g], sg = M.segs[g * M.max_segs + seg];
    const int bad = *wide, skip = A.skip ? *A.skip : 0;
    if (bad || skip || seg >= G.w || strip >= js.y) return;  // uniform
    const int j8 = 8 * (js.x + strip), orient = G.z, NA = G.y, N = kWin * NA;
    const int *shear = M.shear + (size_t)g * M.lblocks;
    const int yb = blockIdx.y * (MT * 128);

    if (tid < 2) s_any[tid] = 0u;
    __syncthreads();
    if (warp < 8) {
        // lines of the segment: warp = line within its block, lanes = blocks
        for (int l0 = 0; l0 < sg.y - sg.x; l0 += 32) {
            const int i = l0 + lane;
            bool any = false;
            if (i < sg.y - sg.x) {
                const int P0 = j8 + shear[sg.x + i];
                int st, lo, hi;
                line_info(A, orient, 8 * (sg.x + i) + warp, st, lo, hi);
                const int first = max(P0, lo) - P0, last = min(P0 + 7, hi) - P0;
                any = first <= last;
                s_ray[i][warp] = any ? st + P0 - lo : 0;
                s_px[i][warp] = any ? (unsigned short)(first | last << 8) : (unsigned short)255;
            }
            const unsigned m = __ballot_sync(0xffffffffu, any);
            if (lane == 0 && m) atomicOr(&s_any[l0 >> 5], m);
        }
    } else if (warp < 16) {
        // window of an angle: one bin below the lowest centre bin of the
        // segment's blocks (all of them, so that strips three apart differ by
        // at least 16)
        if (warp - 8 < NA) {
            const AngleParams ap = A.ang[G.x + warp - 8];
            const float ca = orient ? ap.s : ap.c, cl = orient ? ap.c : ap.s, r = A.r_hi + A.r_lo;
            float mn = 1e30f;
            for (int lb = sg.x + lane; lb < sg.y; lb += 32)
                mn = fminf(mn, ((float)(j8 + shear[lb]) - r) * ca + ((float)(8 * lb) - r) * cl);
            for (int o = 16; o > 0; o >>= 1) mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
            mn += fminf(0.f, 7.f * ca) + fminf(0.f, 7.f * cl) + r;
            if (lane == 0) s_base[warp - 8] = (int)floorf(mn + 0.49f) - 1;
        }
    } else if (warp == kMmaWarp && lane == 0) {
        for (int s = 0; s < C::STAGES; s++) {
            for (int i = 0; i < C::NSUB; i++) {
                umma::mbar_init(&xfull[s][i], 1);
                umma::mbar_init(&xempty[s][i], 1);
            }
            umma::mbar_init(&bfull[s], kBuilders);
            umma::mbar_init(&bempty[s], 1);
        }
        for (int b = 0; b < 2; b++) {
            umma::mbar_init(&accfull[b], 1);
            umma::mbar_init(&accfree[b], kTakers);
        }
        umma::mbar_init(&drained, 1);
        umma::mbar_fence_init();
    }
    __syncthreads();
    // the line blocks that hold rays of this strip, in order
    const unsigned any0 = s_any[0], any1 = s_any[1];
    const int nb = __popc(any0) + __popc(any1);
    if (nb == 0) return;  // uniform
    if (tid < kSegBlocks) {
        const unsigned m = tid < 32 ? any0 : any1, bit = 1u << (tid & 31);
        if (m & bit) blist[(tid < 32 ? 0 : __popc(any0)) + __popc(m & (bit - 1u))] = (short)tid;
    }
    if (warp == kLoadWarp) {
        umma::tmem_alloc(&tmem_base, C::COLS);
        umma::tmem_relinquish();
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = umma::uniform(tmem_base);
    const uint32_t raw = umma::smem_addr(sm_raw);
    unsigned char *sm = sm_raw + ((1024u - (raw & 1023u)) & 1023u);

    if (warp >= kLoadWarp) {
        regs_dec<C::REGS_LOW>();
        if (warp == kLoadWarp) {
            // ---- loads (pixels outside the disk or the image are zeros)
            if (lane == 0) {
                bool ok = true;
                int it = 0, i = 0;
                for (; it < nb && ok; it += ok) {
                    const int s = it % C::STAGES, lb = sg.x + blist[it], P0 = j8 + shear[lb];
                    const int ix = orient ? 8 * lb : P0, iz = orient ? P0 : 8 * lb;
#pragma unroll 1
                    for (i = 0; i < C::NSUB; i++) {
                        if (it >= C::STAGES)
                            ok = umma::mbar_wait(&xempty[s][i], (uint32_t)(it / C::STAGES - 1) & 1u,
                                                 kMmaWait);
                        if (!ok) break;
                        umma::mbar_arrive_expect_tx(&xfull[s][i], (uint32_t)C::SUB);
                        unsigned char *d = sm + (size_t)s * C::STAGE + i * C::SUB;
                        const int y = yb + 128 * (i >> 1);
                        umma::tma_load_4d(d, &tmx, y, ix, iz, 1 - (i & 1), &xfull[s][i]);
                        umma::tma_load_4d(d + 8192, &tmx, y + 64, ix, iz, 1 - (i & 1), &xfull[s][i]);
                    }
                }
                if (!ok) {
                    atomicOr(A.err, 16);
                    // copies in flight: the last line blocks' and the first i of this one's
                    for (int u = max(0, it - C::STAGES); u <= it; u++)
                        for (int j = 0; j < (u < it ? C::NSUB : i); j++)
                            umma::mbar_wait(&xfull[u % C::STAGES][j], (uint32_t)(u / C::STAGES) & 1u,
                                            kMmaWait);
                }
            }
        } else if (warp == kMmaWarp) {
            // ---- MMAs: low-order products first (their sums are small), then
            // hi*hi: the large sum is rounded toward zero four times only
            const uint32_t idesc = idesc_f16(N), kb = (uint32_t)(N / 8) * 128u;
            const uint64_t bk = 2 * kb / 16, bl = 8 * kb / 16;
            constexpr uint64_t AK = 2048 / 16;
            bool ok = true;
            for (int it = 0; it < nb && ok; it++) {
                const int s = it % C::STAGES, b = it & 1;
                const uint32_t ph = (uint32_t)(it / C::STAGES) & 1u;
                ok = umma::mbar_wait_warp(&bfull[s], ph, kMmaWait) &&
                     (it < 2 ||
                      umma::mbar_wait_warp(&accfree[b], (uint32_t)(it / 2 - 1) & 1u, kMmaWait));
                const uint32_t x = umma::smem_addr(sm) + (uint32_t)(s * C::STAGE);
                const uint64_t bd = desc_mn(x + C::X, 128, kb);
#pragma unroll
                for (int mt = 0; mt < MT; mt++) {
                    const uint32_t d = tmem + (uint32_t)((b * MT + mt) * 128);
                    const uint64_t al = desc_mn_sw128(x + 2 * mt * C::SUB, 8192, 1024);
                    const uint64_t ah = desc_mn_sw128(x + (2 * mt + 1) * C::SUB, 8192, 1024);
                    ok = ok && umma::mbar_wait_warp(&xfull[s][2 * mt], ph, kMmaWait);
                    if (!ok) break;
                    umma::fence_after_sync();
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        umma::mma_f16_warp(d, al + k * AK, bd + k * bk, idesc, k > 0 ? 1u : 0u);
                    umma::mma_commit_warp(&xempty[s][2 * mt]);
                    ok = umma::mbar_wait_warp(&xfull[s][2 * mt + 1], ph, kMmaWait);
                    if (!ok) break;
                    umma::fence_after_sync();
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        umma::mma_f16_warp(d, ah + k * AK, bd + bl + k * bk, idesc, 1u);
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        if (k == 0)
                            umma::mma_f16_warp_scaled<kLowBits>(d, ah, bd, idesc);
                        else
                            umma::mma_f16_warp(d, ah + k * AK, bd + k * bk, idesc, 1u);
                    umma::mma_commit_warp(&xempty[s][2 * mt + 1]);
                }
                if (!ok) break;
                umma::mma_commit_warp(&bempty[s]);
                umma::mma_commit_warp(&accfull[b]);
            }
            if (!ok) {
                if (lane == 0) atomicOr(A.err, 16);
                umma::mma_drain_warp(&drained, kMmaWait);  // half a block of rays, uncommitted
            }
        }
        __syncwarp();
    } else if (warp >= kTakers) {
        // ---- weights: one pixel (row, column) of the block, angles a4 and a4 + 4
        regs_dec<C::REGS_LOW>();
        const int row = warp - kTakers, col = lane & 7, a4 = lane >> 3, kb = N / 8 * 128;
        const int line = orient ? col : row, px = orient ? row : col;
        const uint4 *tp[2];
        int base[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int ai = a4 + 4 * h;
            const int slot = ai < NA ? M.slots[G.x + ai] & INT_MAX : 0;
            base[h] = ai < NA ? s_base[ai] + 1 : 0;
            tp[h] = M.taps ? M.taps + (size_t)(slot >> 2) * A.nrays * kGroupAngles + (slot & 3) : nullptr;
        }
        // packed taps of block `it`
        auto fetch = [&](int it, uint4 (&e)[2]) {
            e[0] = make_uint4((unsigned)base[0], 0u, 0u, 0u);  // no ray: zero weights
            e[1] = make_uint4((unsigned)base[1], 0u, 0u, 0u);
            if (it >= nb) return;
            const int lb = blist[it];
            const int ray = s_ray[lb][line] + px, range = s_px[lb][line];
            if (px < (range & 255) || px > range >> 8) return;
#pragma unroll
            for (int h = 0; h < 2; h++)
                if (a4 + 4 * h < NA)
                    e[h] = M.taps ? __ldg(tp[h] + (size_t)ray * kGroupAngles)
                                  : pack_taps(ray_taps<W>(A.ray[orient ? A.kinv[ray] : ray],
                                                          A.ang[G.x + a4 + 4 * h], A.r_hi, A.r_lo));
        };
        bool ok = true;
        auto build = [&](int it, const uint4 (&e)[2]) {
            const int s = it % C::STAGES;
            if (it >= C::STAGES)
                ok = __all_sync(0xffffffffu, umma::mbar_wait(&bempty[s],
                                                             (uint32_t)(it / C::STAGES - 1) & 1u, kMmaWait));
            if (!ok) return;
            unsigned char *d = sm + (size_t)s * C::STAGE + C::X + row * kb + a4 * 256 + col * 16;
#pragma unroll
            for (int h = 0; h < 2; h++)
                if (a4 + 4 * h < NA) {
                    int p = (int)e[h].x - base[h];
                    if ((unsigned)p > (unsigned)kSpread) {
                        atomicOr(A.err, 1);  // outside the window: the segments rule it out
                        p = 0;
                    }
                    store_rows(d + h * 1024, 8 * kb, p, e[h]);
                }
            umma::fence_async_smem();
            __syncwarp();
            if (lane == 0) umma::mbar_arrive(&bfull[s]);
        };
        // two sets of taps in flight (a copy from one to the other would wait for it)
        uint4 e0[2], e1[2];
        fetch(0, e0);
        fetch(1, e1);
        for (int it = 0; it < nb && ok; it += 2) {
            build(it, e0);
            fetch(it + 2, e0);
            if (it + 1 < nb && ok) {
                build(it + 1, e1);
                fetch(it + 3, e1);
            }
        }
        if (!ok && lane == 0) atomicOr(A.err, 16);
    } else {
        // ---- sums: TMEM lanes 32 quarter.., M tile mt, columns c0 .. c0 + ACC
        regs_inc<C::REGS_TAKE>();
        const int quarter = warp & 3, mt = MT == 2 ? warp >> 2 : 0, c0 = MT == 2 ? 0 : (warp >> 2) * C::ACC;
        float acc[C::ACC];
#pragma unroll
        for (int i = 0; i < C::ACC; i++) acc[i] = 0.f;
        bool ok = true;
        for (int it = 0; it < nb; it++) {
            const int b = it & 1;
            ok = __all_sync(0xffffffffu,
                            umma::mbar_wait(&accfull[b], (uint32_t)(it / 2) & 1u, kMmaWait));
            if (!ok) break;
            umma::fence_after_sync();
            const uint32_t col = tmem + ((uint32_t)(32 * quarter) << 16) +
                                 (uint32_t)((b * MT + mt) * 128 + c0);
#pragma unroll
            for (int c = 0; c < C::ACC / 16; c++)
                if (c0 + c * 16 < N) {
                    float v[16];
                    umma::tmem_ld16(col + 16 * c, v);
#pragma unroll
                    for (int i = 0; i < 16; i++) acc[16 * c + i] += v[i];
                }
            umma::fence_before_sync();
            __syncwarp();
            if (lane == 0) umma::mbar_arrive(&accfree[b]);
        }
        if (!ok && lane == 0) atomicOr(A.err, 16);
        const int y = yb + mt * 128 + quarter * 32 + lane;
        if (ok && y < A.ys) {
            const float inv = pow2f(-half_shift(maxb[y])) * (1.f / kWeightScale);
#pragma unroll
            for (int c = 0; c < C::ACC / 16; c++) {
                const int an = c0 / 16 + c;
                if (an < NA) {
                    const int b0 = s_base[an];
                    float *qa = q + ((size_t)(G.x + an) * A.nx) * A.ys + y;
                    // one add per bin and launch: the order is the launches'
#pragma unroll
                    for (int i = 0; i < 16; i++)
                        if ((unsigned)(b0 + i) < (unsigned)A.nx)
                            atomicAdd(qa + (size_t)(b0 + i) * A.ys, acc[16 * c + i] * inv);
                }
            }
        }
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == kLoadWarp) umma::tmem_dealloc(tmem, C::COLS);
}

// ---------------------------------------------------------------------------
// Back projection  g[k][y] = sum_a sum_j w_j(k, a) s[a][b(k, a) + j][y].
//   D[y][k] += sum over a window of 16 bins of S[y][b] W[b][k]:
//   M = 128 slices, N = 64 rays (8 x 8 pixels), K = 16 bins, two angles per set of
// sums in TMEM.  A block owns 16 x 16 pixels (four such sub-blocks) x 128 slices
// and runs over the angles; per angle the sinogram's 32 bins from the lowest
// window on are loaded once, and each sub-block's window is an offset into them.

constexpr int kFoot = 32;  // bins loaded per angle: four windows of 16 within 29 bins
struct BpMma {
    static constexpr int PART = kFoot * 16 * 16;     // [16 slice groups][32 bins][8 slices]
    static constexpr int SUBW = 2048;                // 64 rays x 16 bins
    static constexpr int A = 4 * PART;               // [angle][part]
    static constexpr int B = 16 * SUBW;              // [angle][part][sub-block]
    static constexpr int STAGE = A + B;
    static constexpr int STAGES = 3;
    static constexpr uint32_t COLS = 512;            // two sets of 4 x 64 columns
    static constexpr int MAX_NA = 4096;              // angles: their windows and slots, 8 bytes each
    // of the launch's 61440 registers: 12 warps x 32 x 40 + 8 x 32 x 176 = 60416
    static constexpr int REGS_LOW = 40, REGS_TAKE = 176;
    static size_t smem(int na) { return (size_t)STAGES * STAGE + 8 * (size_t)(na + 2) + 1024; }
};

// First bin of the windows of the tile's four sub-blocks at one angle (one below
// the lowest centre bin): the tile's lowest and the others' distances from it, at
// most 8 (|cos| + |sin|) < 12 bins, as (lowest + 64) << 16 | 4 bits each.
__device__ __forceinline__ unsigned bp_windows(const AngleParams &ap, float r, int x0, int z0) {
    int w[4];
    const float lo = fminf(0.f, 7.f * ap.c) + fminf(0.f, 7.f * ap.s) + r + 0.49f;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float v = __fadd_rn(__fadd_rn(__fmul_rn((float)(x0 + 8 * (i & 1)) - r, ap.c),
                                            __fmul_rn((float)(z0 + 8 * (i >> 1)) - r, ap.s)), lo);
        w[i] = (int)floorf(v) - 1;
    }
    const int f = min(min(w[0], w[1]), min(w[2], w[3]));
    return (unsigned)(f + 64) << 16 | (unsigned)(w[0] - f) | (unsigned)(w[1] - f) << 4 |
           (unsigned)(w[2] - f) << 8 | (unsigned)(w[3] - f) << 12;
}

// Pairs of FP32 numbers.
__device__ __forceinline__ unsigned long long pair(uint32_t a, uint32_t b) {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};\n" : "=l"(v) : "r"(a), "r"(b));
    return v;
}
__device__ __forceinline__ void unpair(unsigned long long v, uint32_t &a, uint32_t &b) {
    asm("mov.b64 {%0, %1}, %2;\n" : "=r"(a), "=r"(b) : "l"(v));
}
// Eight sums in step (the steps of one addition wait for one another):
// acc += v scale; v = what the addition rounded away (exact while |acc| >= |v scale|).
__device__ __forceinline__ void two_sum(unsigned long long *acc, uint32_t *va, unsigned long long scale) {
    unsigned long long v[4], t[4];
#pragma unroll
    for (int i = 0; i < 4; i++) v[i] = pair(va[2 * i], va[2 * i + 1]);
#pragma unroll
    for (int i = 0; i < 4; i++)
        asm volatile("fma.rn.f32x2 %0, %1, %3, %2;\n" : "=l"(t[i]) : "l"(v[i]), "l"(acc[i]), "l"(scale));
#pragma unroll
    for (int i = 0; i < 4; i++) asm volatile("sub.rn.f32x2 %0, %0, %1;\n" : "+l"(acc[i]) : "l"(t[i]));
#pragma unroll
    for (int i = 0; i < 4; i++)
        asm volatile("fma.rn.f32x2 %0, %0, %1, %2;\n" : "+l"(v[i]) : "l"(scale), "l"(acc[i]));
#pragma unroll
    for (int i = 0; i < 4; i++) {
        acc[i] = t[i];
        unpair(v[i], va[2 * i], va[2 * i + 1]);
    }
}

// Roles as in the forward projector; builders: warp = 4 rows of 8 pixels of a
// sub-block half, lane = pixel, both angles; takers: thread = slice, two
// sub-blocks (128 rays).  The takers hand what each addition rounds away back to
// the set it came from, which starts its next sums with it (times 2^11, as the
// low-order products come first): equal addends, hundreds of them in a flat
// sinogram, would all round the same way (6e-6 of the sum at 1200 angles; 4e-8
// with it, 8e-7 for the FP32 kernels).
//
// What bounds it: two angles' 24 MMAs read 24 x 6 KB of shared memory, 1300
// clocks; they take 2460 alone, 2900 beside the takers' traffic with TMEM.  A
// back projection at 1024^2 x 1200 angles x 512 slices takes 72.4 ms, 209.1 with
// the FP32 kernels as a plan comes (110.7 with tuned shapes).
template <int W>
__global__ void __launch_bounds__(kMmaThreads, 1)
    bp_mma_kernel(OpArgs A, MmaPlan M, const __grid_constant__ CUtensorMap tms, float *__restrict__ g,
                  const unsigned *__restrict__ maxb, const int *__restrict__ wide) {
    using C = BpMma;
    extern __shared__ unsigned char sm_raw[];
    __shared__ __align__(8) uint64_t afull[C::STAGES], bfull[C::STAGES], empty[C::STAGES];
    __shared__ __align__(8) uint64_t accfull[2], accfree[2];
    __shared__ uint32_t tmem_base;
    __shared__ int s_k[256];                // rays of the tile (-1: none), sub-block by sub-block
    const int tid = threadIdx.x, warp = umma::uniform(tid >> 5), lane = tid & 31;
    if ((A.skip && *A.skip) || *wide) return;  // uniform
    const int2 tile = M.tiles[blockIdx.x];
    const int yb = blockIdx.y * 128, na = A.na;
    // this block's pairs of angles: all, or one of two halves
    const int pairs = ((na + 1) / 2 + gridDim.z - 1) / gridDim.z, a_lo = 2 * pairs * blockIdx.z;
    const int ns = min(pairs, (na + 1) / 2 - pairs * (int)blockIdx.z);
    const float r = A.r_hi + A.r_lo;

    if (tid < 256) {
        const int i = tid >> 6, ix = tile.x + 8 * (i & 1) + (tid & 7),
                  iz = tile.y + 8 * (i >> 1) + ((tid >> 3) & 7);
        int k = -1;
        if (iz < A.nx) {
            const RowInfo ri = A.rows[iz];
            if (ix >= ri.lo && ix <= ri.hi) k = ri.start + ix - ri.lo;
        }
        s_k[tid] = k;
    }
    if (warp == kLoadWarp) {
        umma::tmem_alloc(&tmem_base, C::COLS);
        umma::tmem_relinquish();
    }
    if (warp == kMmaWarp && lane == 0) {
        for (int s = 0; s < C::STAGES; s++) {
            umma::mbar_init(&afull[s], 1);
            umma::mbar_init(&bfull[s], kBuilders);
            umma::mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; b++) {
            umma::mbar_init(&accfull[b], 1);
            umma::mbar_init(&accfree[b], kTakers);
        }
        umma::mbar_fence_init();
    }
    const uint32_t raw = umma::smem_addr(sm_raw);
    unsigned char *sm = sm_raw + ((1024u - (raw & 1023u)) & 1023u);
    // per angle: windows, place in the taps table (the pair after the last: unused)
    uint2 *s_ang = reinterpret_cast<uint2 *>(sm + C::STAGES * C::STAGE);
    for (int a = tid; a < na; a += kMmaThreads)
        s_ang[a] = make_uint2(bp_windows(A.ang[a], r, tile.x, tile.y), (unsigned)M.slots[a]);
    if (tid == 0) s_ang[na] = s_ang[na + 1] = make_uint2(64u << 16, 0u);
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = umma::uniform(tmem_base);

    if (warp >= kLoadWarp) {
        regs_dec<C::REGS_LOW>();
        if (warp == kLoadWarp && lane == 0) {
            bool ok = true;
            int it = 0;
            for (; it < ns && ok; it++) {
                const int s = it % C::STAGES, a = a_lo + 2 * it, n = min(2, na - a);
                if (it >= C::STAGES)
                    ok = umma::mbar_wait(&empty[s], (uint32_t)(it / C::STAGES - 1) & 1u, kMmaWait);
                if (!ok) break;
                umma::mbar_arrive_expect_tx(&afull[s], (uint32_t)(2 * n * C::PART));
                for (int i = 0; i < n; i++) {
                    const int f = (int)(s_ang[a + i].x >> 16) - 64;
                    unsigned char *d = sm + (size_t)s * C::STAGE + 2 * i * C::PART;
                    umma::tma_load_4d(d, &tms, 8 * f, yb / 8, a + i, 0, &afull[s]);
                    umma::tma_load_4d(d + C::PART, &tms, 8 * f, yb / 8, a + i, 1, &afull[s]);
                }
            }
            if (!ok) {
                atomicOr(A.err, 16);
                umma::ring_drain(afull, C::STAGES, it, kMmaWait);
            }
        } else if (warp == kMmaWarp) {
            // FP16, A MN-major (bit 15), B K-major, N = 64
            const uint32_t idesc = (1u << 4) | (1u << 15) | (8u << 17) | ((128u >> 4) << 24);
            bool ok = true;
            for (int it = 0; it < ns && ok; it++) {
                const int s = it % C::STAGES, b = it & 1, a0 = a_lo + 2 * it, n = min(2, na - a0);
                const uint32_t ph = (uint32_t)(it / C::STAGES) & 1u;
                const uint32_t win[2] = {umma::uniform(s_ang[a0].x), umma::uniform(s_ang[a0 + 1].x)};
                ok = umma::mbar_wait_warp(&bfull[s], ph, kMmaWait) &&
                     umma::mbar_wait_warp(&afull[s], ph, kMmaWait) &&
                     (it < 2 ||
                      umma::mbar_wait_warp(&accfree[b], (uint32_t)(it / 2 - 1) & 1u, kMmaWait));
                if (!ok) break;
                umma::fence_after_sync();
                const uint32_t base = umma::smem_addr(sm) + (uint32_t)(s * C::STAGE);
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const uint32_t d = tmem + (uint32_t)(b * 256 + q * 64);
                    // the low-order products of both angles, then hi*hi
#pragma unroll
                    for (int t = 0; t < 2; t++)
#pragma unroll
                        for (int i = 0; i < 2; i++) {
                            if (i >= n) break;
                            const uint32_t a =
                                base + (uint32_t)(2 * i * C::PART) + (win[i] >> (4 * q) & 15u) * 16u;
                            const uint32_t w = base + (uint32_t)(C::A + (8 * i + q) * C::SUBW);
                            const uint64_t ah = desc_mn(a, kFoot * 16, 128);
                            const uint64_t al = desc_mn(a + C::PART, kFoot * 16, 128);
                            const uint64_t wh = umma::smem_desc(w, 128, 256);
                            const uint64_t wl = umma::smem_desc(w + 4 * C::SUBW, 128, 256);
                            if (t == 0) {
                                umma::mma_f16_warp(d, al, wh, idesc, i > 0 || it > 1 ? 1u : 0u);
                                umma::mma_f16_warp(d, ah, wl, idesc, 1u);
                            } else if (i == 0) {
                                umma::mma_f16_warp_scaled<kLowBits>(d, ah, wh, idesc);
                            } else {
                                umma::mma_f16_warp(d, ah, wh, idesc, 1u);
                            }
                        }
                }
                umma::mma_commit_warp(&empty[s]);
                umma::mma_commit_warp(&accfull[b]);
            }
            // (the takers wait for every set of MMAs issued, each of which is committed)
            if (!ok && lane == 0) atomicOr(A.err, 16);
        }
        __syncwarp();
    } else if (warp >= kTakers) {
        regs_dec<C::REGS_LOW>();
        const int t = tid - 32 * kTakers, q = t >> 6, k = s_k[t];
        const int ix = tile.x + 8 * (q & 1) + (t & 7), iz = tile.y + 8 * (q >> 1) + ((t >> 3) & 7);
        int kc = -1;  // the ray in column-major order (the taps of column sweeps)
        if (k >= 0) {
            const ColInfo ci = A.cols[ix];
            kc = ci.start + iz - ci.lo;
        }
        auto fetch = [&](int it, uint4 (&e)[2]) {
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int a = a_lo + 2 * it + i;
                e[i] = make_uint4(0u, 0u, 0u, 0u);  // no ray: zero weights
                if (it >= ns || a >= na || k < 0) continue;
                if (M.taps) {
                    const int slot = (int)s_ang[a].y;
                    e[i] = __ldg(M.taps + ((size_t)((slot & INT_MAX) >> 2) * A.nrays + (slot < 0 ? kc : k)) *
                                              kGroupAngles + (slot & 3));
                } else {
                    e[i] = pack_taps(ray_taps<W>(A.ray[k], A.ang[a], A.r_hi, A.r_lo));
                }
            }
        };
        bool ok = true;
        auto build = [&](int it, const uint4 (&e)[2]) {
            const int s = it % C::STAGES;
            if (it >= C::STAGES)
                ok = __all_sync(0xffffffffu, umma::mbar_wait(&empty[s],
                                                             (uint32_t)(it / C::STAGES - 1) & 1u, kMmaWait));
            if (!ok) return;
            unsigned char *d = sm + (size_t)s * C::STAGE + C::A + q * C::SUBW + ((t >> 3) & 7) * 256 + (t & 7) * 16;
#pragma unroll
            for (int i = 0; i < 2; i++) {
                if (a_lo + 2 * it + i >= na) break;
                const unsigned win = s_ang[a_lo + 2 * it + i].x;
                int p = (int)e[i].x + 63 - (int)((win >> 16) + (win >> (4 * q) & 15u));
                if (k < 0) p = 0;
                if ((unsigned)p > (unsigned)kSpread) {
                    atomicOr(A.err, 2);  // outside the window: cannot happen
                    p = 0;
                }
                store_rows(d + i * 8 * C::SUBW, 4 * C::SUBW, p, e[i]);
            }
            umma::fence_async_smem();
            __syncwarp();
            if (lane == 0) umma::mbar_arrive(&bfull[s]);
        };
        uint4 e0[2], e1[2];
        fetch(0, e0);
        fetch(1, e1);
        for (int it = 0; it < ns && ok; it += 2) {
            build(it, e0);
            fetch(it + 2, e0);
            if (it + 1 < ns && ok) {
                build(it + 1, e1);
                fetch(it + 3, e1);
            }
        }
        if (!ok && lane == 0) atomicOr(A.err, 16);
    } else {
        regs_inc<C::REGS_TAKE>();
        const int quarter = warp & 3, half = warp >> 2;
        unsigned long long acc[64];
#pragma unroll
        for (int i = 0; i < 64; i++) acc[i] = 0ull;
        const unsigned long long scale = pair(__float_as_uint(kLowScale), __float_as_uint(kLowScale));
        bool ok = true;
        for (int it = 0; it < ns; it++) {
            const int b = it & 1;
            ok = __all_sync(0xffffffffu,
                            umma::mbar_wait(&accfull[b], (uint32_t)(it / 2) & 1u, kMmaWait));
            if (!ok) break;
            umma::fence_after_sync();
            const uint32_t col = tmem + ((uint32_t)(32 * quarter) << 16) + (uint32_t)(b * 256 + half * 128);
#pragma unroll
            for (int c = 0; c < 8; c++) {
                uint32_t v[16];
                umma::tmem_ld16(col + 16 * c, v);
#pragma unroll
                for (int i = 0; i < 2; i++) two_sum(acc + 8 * c + 4 * i, v + 8 * i, scale);
                umma::tmem_st16(col + 16 * c, v);
            }
            umma::tmem_wait_st();
            umma::fence_before_sync();
            __syncwarp();
            if (lane == 0) umma::mbar_arrive(&accfree[b]);
        }
        if (!ok && lane == 0) atomicOr(A.err, 16);
        const int y = yb + quarter * 32 + lane;
        if (ok && y < A.ys) {
            const float inv = pow2f(-half_shift(maxb[y])) * (1.f / (kWeightScale * kLowScale));
#pragma unroll
            for (int i = 0; i < 64; i++) {
                uint32_t va, vb;
                unpair(acc[i], va, vb);
                const int ka = s_k[half * 128 + 2 * i], kb = s_k[half * 128 + 2 * i + 1];
                float *pa = g + (size_t)ka * A.ys + y, *pb = g + (size_t)kb * A.ys + y;
                const float fa = __uint_as_float(va) * inv, fb = __uint_as_float(vb) * inv;
                if (gridDim.z > 1) {  // two halves into zeros: the order does not matter
                    if (ka >= 0) atomicAdd(pa, fa);
                    if (kb >= 0) atomicAdd(pb, fb);
                } else {
                    if (ka >= 0) *pa = fa;
                    if (kb >= 0) *pb = fb;
                }
            }
        }
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == kLoadWarp) umma::tmem_dealloc(tmem, C::COLS);
}

// ---------------------------------------------------------------------------
// Plan: groups, strips and segments.

struct Seg {
    std::vector<int2> segs;
    std::vector<int> shear;
};

// Segments of the angles [a0, a0 + n): line blocks over which
//   shear(lb) ca + 8 lb cl
// varies by at most 12.9 - 7 (|ca| + |cl|) bins for every angle (a block's own
// pixels span 7 (|ca| + |cl|) <= 9.9; centre bins then take at most 14
// neighbouring values, slots 0 .. 13 of the window).
Seg make_segments(const std::vector<AngleParams> &ang, int a0, int n, int orient, int nlb, double r) {
    Seg s;
    const AngleParams &m = ang[a0 + n / 2];
    const double cam = orient ? m.s : m.c, clm = orient ? m.c : m.s;
    s.shear.resize(nlb);
    for (int lb = 0; lb < nlb; lb++)
        s.shear[lb] = (int)std::lround(-(8.0 * lb + 3.5 - r) * clm / cam);
    std::vector<double> lo(n), hi(n);
    for (int lb = 0, first = 0; lb <= nlb; lb++) {
        bool fits = lb < nlb && lb - first < kSegBlocks;
        for (int i = 0; fits && i < n; i++) {
            const double ca = orient ? ang[a0 + i].s : ang[a0 + i].c;
            const double cl = orient ? ang[a0 + i].c : ang[a0 + i].s;
            const double v = s.shear[lb] * ca + 8.0 * lb * cl;
            const double l = lb == first ? v : std::min(lo[i], v), h = lb == first ? v : std::max(hi[i], v);
            if (h - l > 12.9 - 7.0 * (std::fabs(ca) + std::fabs(cl))) fits = false;
            else lo[i] = l, hi[i] = h;
        }
        if (!fits) {
            s.segs.push_back(make_int2(first, lb));
            if (lb == nlb) break;
            first = lb;
            lb--;  // this line block starts the next segment
        }
    }
    return s;
}

template <typename T>
int upload(T **d, const std::vector<T> &h) {
    ARECGB_CUDA(dev_malloc(d, sizeof(T) * std::max<size_t>(h.size(), 1)));
    ARECGB_CUDA(cudaMemcpy(*d, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice));
    return 0;
}

}  // namespace

// Line blocks per segment a group of angles keeps on average, or it takes fewer
// angles: a segment's end costs about as much as three line blocks.  With 3, 6,
// 10 and 16: 58.2, 55.2, 54.7 and 55.6 ms for 50 SIRT iterations at 256^2 x 180
// x 64, 28.5, 28.5, 28.3 and 28.8 ms for CGLS at 401^2 x 300 x 75 (Kaiser-Bessel).
static const int kMinBlocks = 10;

// 2 (every projection of the plan) from 32 bins, 48 slices and 64 angles on, or
// 4 million values in a volume: a back projection of a small volume is a chain over the
// angles, 0.6 us each and 25 us of conversions and launches here against 1.1 us each
// (65^2 x 90 x 64: 0.078 against 0.093 ms, forward 0.091 against 0.139; 256^2 x 180 x
// 64: 0.26 against 0.58, forward 0.51 against 1.03; the FP32 kernels with tables).
// 1 (all but CGLS) with fewer slices and 2.3 million rays and angles (twice that and
// more for Kaiser-Bessel, whose taps cost more to compute): 160^2 x 90 x 16 0.094
// against 0.107 ms, forward 0.20 against 0.36; 1024^2 x 600 x 8 10.7 against 17.8,
// forward 11.5 against 36.6; at 96^2 x 24 x 8 it would be 0.043 against 0.029.  A long
// CGLS solve amplifies rounding (every float solve leaves FP64's trajectory after six
// to eight steps, the reference's too).  With fewer than 48 slices it stays on the FP32
// kernels, which sum in the reference's order, and small solves keep its residual
// trace; that is a choice, not a matter of time.  From 48 slices on it ends 2 to 10
// times nearer FP64 here.  4096 angles fill the back projector's table.
int mma_takes(int weighting, int nx, int ys, int na) {
    if (weighting == ARECGB_LIN || nx < 32 || na > BpMma::MAX_NA) return 0;
    const double px = (double)nx * nx;
    if (ys >= 48) return na >= 64 || px * ys >= 4e6 ? 2 : 0;
    return px * na >= (weighting == ARECGB_KB ? 6e6 : 2.3e6) ? 1 : 0;
}

int mma_plan_create(Plan *p, const std::vector<int4> &g4, const std::vector<AngleParams> &ang,
                    const std::vector<RowInfo> &rows, const std::vector<ColInfo> &cols, bool spare) {
    const int use = mma_takes(p->weighting, p->nx, p->ys, p->na);
    if (!use) return 0;
    for (const AngleParams &a : ang)
        if (!std::isfinite(a.c) || !std::isfinite(a.s)) return 0;  // no strips to follow
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) return 0;
    const size_t work = mma_work_bytes(p->nx, p->na, p->ys);
    if (spare && (double)work > 0.4 * (double)free_b) return 0;
    // a solve must still fit beside them: the caller's volume and sinogram and CGLS's three
    // and two; only these where the caller budgets its memory (spare is false)
    const size_t extra = spare ? 1 : 0;
    if (work + sizeof(float) * ((3 + extra) * vol_floats(p) + (2 + extra) * sin_floats(p)) > free_b) return 0;
    const int nlb = (p->nx + 7) / 8;
    std::vector<int4> groups;
    std::vector<int2> strips;
    std::vector<Seg> segs;
    std::vector<int> slots(p->na);
    for (size_t g = 0; g < g4.size(); g++)
        for (int k = 0; k < g4[g].y; k++) slots[g4[g].x + k] = ((int)g * kGroupAngles + k) | (g4[g].z ? INT_MIN : 0);
    for (int a = 0; a < p->na;) {
        const int o = ang[a].orient;
        int n = 1;
        while (n < 8 && a + n < p->na && ang[a + n].orient == o) n++;
        Seg s = make_segments(ang, a, n, o, nlb, p->radius);
        while (n > 1 && (int)s.segs.size() * kMinBlocks > nlb)
            s = make_segments(ang, a, --n, o, nlb, p->radius);
        int jlo = INT_MAX, jhi = INT_MIN;
        for (int lb = 0; lb < nlb; lb++)
            for (int l = 8 * lb; l < std::min(p->nx, 8 * lb + 8); l++) {
                const int lo = o ? cols[l].lo : rows[l].lo, hi = o ? cols[l].hi : rows[l].hi;
                if (lo > hi) continue;
                jlo = std::min(jlo, (int)std::floor((lo - s.shear[lb]) / 8.0));
                jhi = std::max(jhi, (int)std::floor((hi - s.shear[lb]) / 8.0));
            }
        groups.push_back(make_int4(a, n, o, (int)s.segs.size()));
        strips.push_back(make_int2(jlo, jhi - jlo + 1));
        segs.push_back(std::move(s));
        a += n;
    }
    const int ng = (int)groups.size();
    int ms = 0, mstrips = 0;
    for (int g = 0; g < ng; g++) {
        ms = std::max(ms, (int)segs[g].segs.size());
        mstrips = std::max(mstrips, strips[g].y);
    }
    std::vector<int2> segv((size_t)ng * ms, make_int2(0, 0));
    std::vector<int> shear((size_t)ng * nlb);
    for (int g = 0; g < ng; g++) {
        std::copy(segs[g].segs.begin(), segs[g].segs.end(), segv.begin() + (size_t)g * ms);
        std::copy(segs[g].shear.begin(), segs[g].shear.end(), shear.begin() + (size_t)g * nlb);
    }
    std::vector<int2> tiles;  // 16 x 16 pixels holding at least one ray
    for (int z = 0; z < p->nx; z += 16)
        for (int x = 0; x < p->nx; x += 16) {
            bool any = false;
            for (int iz = z; iz < std::min(p->nx, z + 16) && !any; iz++)
                any = rows[iz].lo <= rows[iz].hi && rows[iz].lo <= x + 15 && rows[iz].hi >= x;
            if (any) tiles.push_back(make_int2(x, z));
        }
    p->m_tiles = (int)tiles.size();
    int rc = upload(&p->d_mgroups, groups);
    if (!rc) rc = upload(&p->d_mtiles, tiles);
    if (!rc) rc = upload(&p->d_mstrips, strips);
    if (!rc) rc = upload(&p->d_msegs, segv);
    if (!rc) rc = upload(&p->d_mshear, shear);
    if (!rc) rc = upload(&p->d_mslots, slots);
    if (rc) return rc;
    p->m_groups = ng;
    p->m_segs = ms;
    p->m_strips = mstrips;
    // per ray its pixel in the image stack
    std::vector<int> pix(p->nrays);
    for (int iz = 0; iz < p->nx; iz++)
        for (int ix = rows[iz].lo; ix <= rows[iz].hi; ix++)
            pix[rows[iz].start + ix - rows[iz].lo] = iz * p->nx + ix;
    if ((rc = upload(&p->d_mpix, pix))) return rc;
    // FP16 pairs of the volume as an image stack (zero outside the disk: never
    // written), and the slices' maxima
    const size_t bytes[2] = {sizeof(float) * (size_t)p->nx * p->nx * p->ys, sizeof(float) * sin_floats(p)};
    for (int d = 0; d < 2; d++) {
        if (dev_malloc(&p->d_half[d], bytes[d]) != cudaSuccess ||
            dev_malloc(&p->d_smax[d], mma_stats_bytes(p->ys)) != cudaSuccess) {
            cudaGetLastError();  // not sticky: run without
            mma_plan_destroy(p);
            return 0;
        }
    }
    ARECGB_CUDA(cudaMemsetAsync(p->d_half[0], 0, bytes[0], p->stream));
    ARECGB_CUDA(cudaStreamSynchronize(p->stream));
    p->mma = use;
    return 0;
}

// The packed taps table (the caller has checked the memory).
int mma_build_taps(Plan *p, const OpArgs &A) {
    const size_t n = (size_t)p->ngroups * p->nrays * kGroupAngles;
    const unsigned blocks = (unsigned)((n + 255) / 256);
    if (p->weighting == ARECGB_KB)
        k_packed_taps<ARECGB_KB><<<blocks, 256, 0, p->stream>>>(A, p->d_ptaps);
    else
        k_packed_taps<ARECGB_SQ><<<blocks, 256, 0, p->stream>>>(A, p->d_ptaps);
    ARECGB_CUDA(cudaGetLastError());
    return 0;
}

void mma_plan_destroy(Plan *p) {
    auto drop = [](auto *&d) {
        cudaFree(d);
        d = nullptr;
    };
    drop(p->d_ptaps);
    drop(p->d_mgroups);
    drop(p->d_mstrips);
    drop(p->d_msegs);
    drop(p->d_mshear);
    drop(p->d_mslots);
    drop(p->d_mpix);
    drop(p->d_mtiles);
    for (int d = 0; d < 2; d++) {
        drop(p->d_half[d]);
        drop(p->d_smax[d]);
    }
    p->mma = 0;
}

static MmaPlan make_plan(const Plan *p) {
    return MmaPlan{p->d_mgroups, p->d_mstrips, p->d_msegs, p->d_mshear, p->d_mslots, p->d_ptaps,
                   p->d_mtiles, p->m_groups, p->m_segs, p->m_strips, (p->nx + 7) / 8};
}

namespace {

// One projection (dir 0 forward, 1 back) on stream st and its operand.
struct Work {
    const Plan *p;
    int dir;
    cudaStream_t st;
    void *half;
    unsigned *smax;
    HalfStats stats;

    Work(const Plan *plan, int d, const MmaOperand &op, cudaStream_t stream)
        : p(plan), dir(d), st(stream), half(op.half), smax(op.stats) {
        stats = {smax, (unsigned long long *)(smax + p->ys), (int *)(smax + 3 * p->ys), p->ys};
    }
};

// Largest magnitude per slice of rows [n][ys], the scores cleared.
int slice_max(const Work &w, const float *v, size_t n, const int *skip) {
    const int ys4 = w.p->ys / 4, nv = std::min(ys4, 256), rb = 256 / nv;
    ARECGB_CUDA(cudaMemsetAsync(w.smax, 0, mma_stats_bytes(w.p->ys), w.st));
    k_slice_max<<<(int)std::min<size_t>(152 * 8, (n + rb - 1) / rb), 256, 16 * nv, w.st>>>(
        (const float4 *)v, n, ys4, w.smax, skip);
    count_launches(1);
    ARECGB_CUDA(cudaGetLastError());
    return 0;
}

// About `blocks` of them, a multiple of `unit`.
unsigned blocks_of(int unit, size_t blocks) {
    return (unsigned)((blocks + unit - 1) / unit * unit);
}
size_t score_bytes(int ys) { return ys <= kScoreShared ? sizeof(int) * ys : 0; }

template <int W, int MT>
int launch_fp_mma(const Work &w, const OpArgs &A, const MmaPlan &M, const CUtensorMap &tx, float *q) {
    if (int rc = set_smem((const void *)fp_mma_kernel<W, MT>, FpMma<MT>::SMEM)) return rc;
    const dim3 grid(M.ngroups * ((M.max_strips + 2) / 3), (A.ys + 128 * MT - 1) / (128 * MT));
    for (int seg = 0; seg < M.max_segs; seg++)
        for (int color = 0; color < 3; color++)
            fp_mma_kernel<W, MT><<<grid, kMmaThreads, FpMma<MT>::SMEM, w.st>>>(A, M, tx, q, w.smax,
                                                                               w.stats.wide, seg, color);
    count_launches(3 * M.max_segs);
    ARECGB_CUDA(cudaGetLastError());
    return 0;
}

// An operand that the pairs cannot hold is projected here, on the FP32 kernels (without
// the plan's tables); for any other n_clear float4 of the output are cleared.  One value
// of 1e12 or an infinity at 512^2 x 360 x 128: 10.8 ms forward and 4.4 back (1.9 and 1.6
// on the tensor cores, 7.0 and 3.2 on the FP32 kernels with tables, as a plan with few
// angles or slices has them); at 1024^2 x 1200 x 512 240 and 146 (44, 73; 160, 209).  A
// kernel of its own that took the rays one by one for each output was 361 and 46 at the
// first size.
int wide_step(const Work &w, OpArgs A, const float *in, float *out, bool back, size_t n_clear) {
    const Plan *p = w.p;
    A.taps = nullptr;
    const auto launch = p->weighting == ARECGB_KB ? launch_wide_kb : launch_wide_sq;
    const int vec = back ? (p->bp_vec ? p->bp_vec : p->vec) : (p->fp_vec ? p->fp_vec : p->vec);
    const WideArgs wa{(const long long *)w.stats.score, w.stats.wide, n_clear};
    const int rc = launch(A, vec, p->ntiles, p->ngroups_o[0], p->fp_band, in, out, back, wa, w.st);
    count_launches(1);
    ARECGB_CUDA(cudaGetLastError());
    return rc ? ARECGB_ERR_ARG : 0;
}

int fp_steps(const Work &w, const OpArgs &A, const float *d_x, float *d_q) {
    const Plan *p = w.p;
    const int ys8 = p->ys / 8;
    const size_t n = p->nrays, total = n * ys8;
    if (int rc = slice_max(w, d_x, n, A.skip)) return rc;
    const int unit = ys8 / std::gcd(ys8, 256);  // blocks whose threads are a multiple of ys8
    k_to_half<<<blocks_of(unit, std::min<size_t>(152 * 4, (total + 255) / 256)), 256, score_bytes(p->ys),
                w.st>>>((const float4 *)d_x, n, ys8, w.stats, p->d_mpix, (size_t)p->nx * p->nx,
                        (uint4 *)w.half, A.skip);
    count_launches(1);
    if (int rc = wide_step(w, A, d_x, d_q, false, sin_floats(p) / 4)) return rc;
    CUtensorMap tx;
    if (!encode_half_map(&tx, w.half, p->ys, p->nx, p->nx, 8, 8)) {
        set_error("forward_project: tensor map encoding failed");
        return ARECGB_ERR_ARG;
    }
    const MmaPlan M = make_plan(p);
    const bool kb = p->weighting == ARECGB_KB;
    if (p->ys > 128)
        return kb ? launch_fp_mma<ARECGB_KB, 2>(w, A, M, tx, d_q) : launch_fp_mma<ARECGB_SQ, 2>(w, A, M, tx, d_q);
    return kb ? launch_fp_mma<ARECGB_KB, 1>(w, A, M, tx, d_q) : launch_fp_mma<ARECGB_SQ, 1>(w, A, M, tx, d_q);
}

template <int W>
int launch_bp_mma(const Work &w, const OpArgs &A, const CUtensorMap &ts, float *g, bool halves) {
    if (int rc = set_smem((const void *)bp_mma_kernel<W>, BpMma::smem(BpMma::MAX_NA))) return rc;
    bp_mma_kernel<W><<<dim3(w.p->m_tiles, (A.ys + 127) / 128, halves ? 2 : 1), kMmaThreads,
                       BpMma::smem(A.na), w.st>>>(
        A, make_plan(w.p), ts, g, w.smax, w.stats.wide);
    count_launches(1);
    ARECGB_CUDA(cudaGetLastError());
    return 0;
}

int bp_steps(const Work &w, const OpArgs &A, const float *d_s, float *d_g) {
    const Plan *p = w.p;
    const int ys8 = p->ys / 8;
    if (int rc = slice_max(w, d_s, (size_t)p->na * p->nx, A.skip)) return rc;
    const int nmb = (ys8 + 3) / 4, unit = nmb / std::gcd(nmb, 8);
    const size_t warps = (size_t)p->na * ((p->nx + 7) / 8) * nmb;
    k_sino_to_half<<<blocks_of(unit, std::min<size_t>(152 * 4, (warps + 7) / 8)), 256, score_bytes(p->ys),
                     w.st>>>((const float4 *)d_s, p->na, p->nx, ys8, w.stats, (uint4 *)w.half, A.skip);
    count_launches(1);
    CUtensorMap ts;
    if (!encode_foot_map(&ts, w.half, p->nx, ys8, p->na, kFoot)) {
        set_error("back_project: tensor map encoding failed");
        return ARECGB_ERR_ARG;
    }
    // Two blocks per tile, half of the angles each, where the SMs' last wave gains: one
    // wave lasts as long as its angles (256^2 x 180 x 64, 208 tiles: two waves of 90
    // pairs or three of 45).
    const int n = p->m_tiles * ((A.ys + 127) / 128);
    const bool halves = A.na >= 32 && 10 * ((2 * n + 151) / 152) < 18 * ((n + 151) / 152);
    if (int rc = wide_step(w, A, d_s, d_g, true, halves ? vol_floats(p) / 4 : 0)) return rc;
    return p->weighting == ARECGB_KB ? launch_bp_mma<ARECGB_KB>(w, A, ts, d_g, halves)
                                     : launch_bp_mma<ARECGB_SQ>(w, A, ts, d_g, halves);
}

}  // namespace

// q = A x.
int forward_project_mma(const Plan *p, const MmaOperand &op, const float *d_x, float *d_q,
                        const int *d_skip, cudaStream_t st) {
    return fp_steps(Work(p, 0, op, st), make_args(p, d_skip), d_x, d_q);
}

// g = A^T s.
int back_project_mma(const Plan *p, const MmaOperand &op, const float *d_s, float *d_g,
                     const int *d_skip, cudaStream_t st) {
    return bp_steps(Work(p, 1, op, st), make_args(p, d_skip), d_s, d_g);
}

// ---------------------------------------------------------------------------
// Operands of captured calls.  A graph's replays are ordered with nothing else, so it
// has memory of its own, which lives as long as it, its clones and its instances (a
// user object they hold).  Allocation nodes would do that too, but not in a graph that
// is cloned, a child of another or instantiated twice.  Calls captured on one stream
// follow one another and share it.
namespace {

struct GraphMemory {
    int device = 0;
    void *ptr = nullptr;
    size_t bytes = 0;
};
// Memory of graphs that are gone.  Never destroyed: graphs may go after this library's
// static objects, at the end of the process.
struct FreeGraphMemory {
    std::mutex mu;
    std::vector<GraphMemory> list;
};
FreeGraphMemory &graph_free() {
    static FreeGraphMemory *f = new FreeGraphMemory;
    return *f;
}

// May not call into CUDA: the memory is taken again, or freed by graph_memory_trim.
void graph_memory_drop(void *m) {
    FreeGraphMemory &f = graph_free();
    std::lock_guard<std::mutex> lk(f.mu);
    f.list.push_back(*static_cast<GraphMemory *>(m));
    delete static_cast<GraphMemory *>(m);
}

// `bytes` held by `graph`, or null.
void *graph_memory(cudaGraph_t graph, size_t bytes) {
    GraphMemory *m = new GraphMemory;
    if (cudaGetDevice(&m->device) == cudaSuccess) {
        FreeGraphMemory &f = graph_free();
        std::lock_guard<std::mutex> lk(f.mu);
        for (size_t i = 0; i < f.list.size() && !m->ptr; i++)
            if (f.list[i].device == m->device && f.list[i].bytes == bytes) {
                *m = f.list[i];
                f.list.erase(f.list.begin() + i);
            }
    }
    if (!m->ptr) {
        m->bytes = bytes;
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;  // this capture is no bar
        const bool relaxed = cudaThreadExchangeStreamCaptureMode(&mode) == cudaSuccess;
        if (!relaxed || dev_malloc(&m->ptr, bytes) != cudaSuccess) m->ptr = nullptr;
        if (relaxed) cudaThreadExchangeStreamCaptureMode(&mode);
    }
    cudaUserObject_t obj = nullptr;
    if (!m->ptr) {
        delete m;
    } else if (cudaUserObjectCreate(&obj, m, graph_memory_drop, 1, cudaUserObjectNoDestructorSync) !=
               cudaSuccess) {
        graph_memory_drop(m);
    } else {
        void *ptr = m->ptr;
        if (cudaGraphRetainUserObject(graph, obj, 1, cudaGraphUserObjectMove) == cudaSuccess) return ptr;
        cudaUserObjectRelease(obj, 1);
    }
    cudaGetLastError();  // not sticky
    return nullptr;
}

}  // namespace

void graph_memory_trim() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return;
    FreeGraphMemory &f = graph_free();
    std::lock_guard<std::mutex> lk(f.mu);
    for (size_t i = f.list.size(); i-- > 0;)
        if (f.list[i].device == dev) {
            cudaFree(f.list[i].ptr);
            f.list.erase(f.list.begin() + i);
        }
}

int mma_operand(const Plan *p, int dir, const int *d_skip, cudaStream_t st, MmaOperand *op) {
    *op = {p->d_half[dir], p->d_smax[dir]};
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    unsigned long long id = 0;
    cudaGraph_t graph = nullptr;
    ARECGB_CUDA(cudaStreamGetCaptureInfo(st, &cap, &id, &graph));
    if (cap == cudaStreamCaptureStatusNone || d_skip) return 0;  // eager, or a solver's (MmaHold)
    std::lock_guard<std::mutex> lk(p->graph_lock);
    const size_t half = sizeof(float) * (dir ? sin_floats(p) : (size_t)p->nx * p->nx * p->ys);
    Plan::GraphOperand &g = p->graph_op[dir];
    if (g.capture != id || g.stream != st || !g.ptr) {
        g.ptr = graph_memory(graph, half + mma_stats_bytes(p->ys));
        g.capture = id;
        g.stream = st;
        if (!g.ptr) {
            *op = {};
            return 0;
        }
        // pixels outside the disk are read and never written
        if (dir == 0) ARECGB_CUDA(cudaMemsetAsync(g.ptr, 0, half, st));
    }
    *op = {g.ptr, (unsigned *)((char *)g.ptr + half)};
    return 0;
}

MmaHold::MmaHold(Plan *const *plans, int n, cudaStream_t s) : st(s) {
    for (int i = 0; i < n; i++)
        if (plans[i]->mma == 2) held.push_back(plans[i]);
    std::sort(held.begin(), held.end());  // one order for all holders
    for (Plan *p : held)
        for (int d = 0; d < 2; d++) {
            p->turn_lock[d].lock();
            cudaStreamWaitEvent(st, p->turn_ev[d], 0);
        }
}

MmaHold::~MmaHold() {
    for (Plan *p : held)
        for (int d = 0; d < 2; d++) {
            cudaEventRecord(p->turn_ev[d], st);
            p->turn_lock[d].unlock();
        }
}

}  // namespace arecgb
