// Projectors on the tensor cores (square-pixel and Kaiser-Bessel weightings):
// shared definitions of arec_project_mma.cu and the projector dispatch.
//
// A projection is a product with a sparse matrix: a ray adds to three bins.
// Taken 8 x 8 pixels at a time the matrix is dense enough for the tensor cores:
// at any angle the 64 rays of a block reach at most 13 neighbouring bins, so
// with windows of 16 bins a block's product with one angle is a 64 x 16 matrix
// per slice, 16/3 of the multiply-adds of the sparse one, at 24 times the FP32
// rate.  Both factors are split into two FP16 numbers each: three products
// hi*hi, hi*lo, lo*hi carry 22 bits.  The tensor core's FP32 accumulation rounds
// toward zero, so a sum stays in TMEM for one block only; FP32 registers take
// it from there with ordinary rounding.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>

#include "arec_internal.cuh"

namespace arecgb {

// FP16 pairs: hi = fp16(v), lo = fp16((v - hi) 2^11), v = the weight times 2^12 or
// the slice's value times 2^half_shift(the slice's largest magnitude).  The low
// halves' own scale (taken back by the MMA that adds hi*hi, D = A B + D 2^-11)
// keeps them normal: 22 bits down to 2^-29 of the slice's largest magnitude, an
// error of 2^-51 of it below.  An operand with a slice that spans more than that
// (see kSmall in arec_project_mma.cu) takes FP32 kernels.
constexpr float kWeightScale = 4096.f;
constexpr int kLowBits = 11;
constexpr float kLowScale = 2048.f;
// So does one with values from 2^40 on, an infinity or a NaN.
constexpr unsigned kWideBits = (127u + 40u) << 23;

__device__ __forceinline__ int half_shift(unsigned max_bits) {
    if (max_bits == 0u) return 0;
    const int e = (int)(max_bits >> 23) - 127;
    return max(-126, min(126, 14 - e));  // |v| 2^shift < 2^15
}
__device__ __forceinline__ float pow2f(int e) { return __uint_as_float((unsigned)(e + 127) << 23); }

// Forward projection groups, strips and segments (see arec_project_mma.cu).
struct MmaPlan {
    const int4 *groups;   // (first angle, angles, orientation, segments)
    const int2 *strips;   // (first strip, strips)
    const int2 *segs;     // [groups][max_segs]: line blocks [first, last)
    const int *shear;     // [groups][lblocks]: the strips' offset in pixels per line block
    const int *slots;     // per angle its place in the taps table: 4 * (4-angle group) + column,
                          // the sign bit set for column sweeps
    const uint4 *taps;    // packed taps (null: computed by the kernel)
    const int2 *tiles;    // back projection: 16 x 16-pixel tiles (first ix, iz)
    int ngroups, max_segs, max_strips, lblocks;
};

// Which of a plan's projections run on the tensor cores (Plan::mma).
int mma_takes(int weighting, int nx, int ys, int na);
// spare: leave the plan to the FP32 kernels (p->mma = 0) when the operands would
// take more than 40 % of the free memory.  It is left to them in any case when
// they cannot be allocated or would leave no room for a solve.
int mma_plan_create(Plan *p, const std::vector<int4> &groups4,
                    const std::vector<AngleParams> &ang, const std::vector<RowInfo> &rows,
                    const std::vector<ColInfo> &cols, bool spare);
struct OpArgs;
int mma_build_taps(Plan *p, const OpArgs &A);
void mma_plan_destroy(Plan *p);
// Memory of one projection: its operand as FP16 pairs and what HalfStats holds.
struct MmaOperand {
    void *half = nullptr;
    unsigned *stats = nullptr;
};
// The operand of a projection (dir 0 forward, 1 back) on stream st: the plan's, or in a
// capture (but a solver's: d_skip) one that the graph holds; half null when there is no
// memory for that, and the call takes the FP32 kernels.
int mma_operand(const Plan *p, int dir, const int *d_skip, cudaStream_t st, MmaOperand *op);
int forward_project_mma(const Plan *p, const MmaOperand &op, const float *d_x, float *d_q,
                        const int *d_skip, cudaStream_t st);
int back_project_mma(const Plan *p, const MmaOperand &op, const float *d_s, float *d_g,
                     const int *d_skip, cudaStream_t st);

// A plan's turns in both directions, held around launches of graphs whose projections
// use its operands.
class MmaHold {
  public:
    MmaHold(Plan *const *plans, int n, cudaStream_t st);
    ~MmaHold();
    MmaHold(const MmaHold &) = delete;
    MmaHold &operator=(const MmaHold &) = delete;

  private:
    std::vector<Plan *> held;
    cudaStream_t st;
};

// Bytes of an operand's maxima and scores, and of both FP16 operands of a plan
// with theirs.
inline size_t mma_stats_bytes(size_t ys) { return sizeof(unsigned) * (3 * ys + 4); }
inline size_t mma_work_bytes(size_t nx, size_t na, size_t ys) {
    return sizeof(float) * (nx * nx * ys + na * nx * ys) + 2 * mma_stats_bytes(ys);
}

}  // namespace arecgb
