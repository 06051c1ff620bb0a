// Arguments the projector kernels share.
#pragma once

#include "arec_internal.cuh"

namespace arecgb {

struct OpArgs {
    const float4 *ray;
    const AngleParams *ang;
    const RowInfo *rows;
    const ColInfo *cols;
    const int4 *groups;
    const int2 *tiles;
    int nx, nrays, ys, na, ngroups;
    float r_hi, r_lo;
    double *partials;
    const int *skip;
    int *err;
    // linear weighting: per angle, the rays grouped by first bin (lin_off
    // [na][nx+2]: bucket j holds the rays whose first bin is j - 1; lin_list
    // [na][nrays]: ray indices, ascending within a bucket)
    const int *lin_off;
    const int *lin_list;
    // optional per-plan tables (null when the plan has none)
    const float4 *taps;  // [ngroups][nrays][4]: ray_taps of each forward-projection angle
                         // group's (up to 4) angles per ray: (iqx, w0, w1, w2)
    const float4 *bpw;   // [ntiles][na][32]: the back projector's plan entries
    const int2 *bpf;     // [ntiles][na]: footprint (first bin, bins) per tile and angle
    const int *kinv;     // column-major ray index -> ray index
};

// What a projection does about an operand that FP16 pairs cannot hold (operand_wide in
// arec_project_impl.cuh): [ys] scores, the flag, float4 of the output to clear otherwise.
struct WideArgs {
    const long long *score;
    int *wide;
    size_t n_clear;
};

inline OpArgs make_args(const Plan *p, const int *skip) {
    OpArgs A;
    A.ray = p->d_ray;
    A.ang = p->d_ang;
    A.rows = p->d_rows;
    A.cols = p->d_cols;
    A.groups = p->d_groups;
    A.tiles = p->d_tiles;
    A.nx = p->nx;
    A.nrays = p->nrays;
    A.ys = p->ys;
    A.na = p->na;
    A.ngroups = p->ngroups;
    A.r_hi = p->r_hi;
    A.r_lo = p->r_lo;
    A.partials = p->d_bp_partials;
    A.skip = skip;
    A.err = p->d_err;
    A.taps = p->d_taps;
    A.bpw = p->d_bpw;
    A.bpf = p->d_bpf;
    A.kinv = p->d_kinv;
    A.lin_off = p->d_lin_off;
    A.lin_list = p->d_lin_list;
    return A;
}

}  // namespace arecgb
