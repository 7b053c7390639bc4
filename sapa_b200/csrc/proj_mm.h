// proj_mm.h — argument records of the kernels in sapa_proj_mm.cu.
#pragma once

#include <cstddef>

#include <cuda_runtime.h>

namespace sapa {
namespace pmm {

constexpr int MAX_PROBLEMS = 3;
constexpr int MAX_GROUPS = 256;
constexpr int MAX_D_NORM = 64;         // rows of W behind a norm that the backward takes

// GroupNorm statistics: partial sums of the slices of every (image, group)
struct StatProblem {
    const void *x;
    double2 *partial;                  // [B * groups][nsplit]
    long long n;                       // elements of a group
    int nsplit, blocks, vec;
};
struct StatList { StatProblem p[MAX_PROBLEMS]; int count; };

// out[b, m, p] = sum_k W[m, k] norm(x)[b, k, p] + bias_m
struct FwdProblem {
    const void *x, *weight, *bias, *gamma, *beta;
    const double2 *partial;            // from the statistics kernel, nullptr: no norm
    float2 *stats;                     // (mean, rstd) per (image, group) for the backward, or nullptr
    void *out;
    long long n;
    float eps;
    int B, M, K, HW, groups, cpg, nsplit, mblocks, pblocks, blocks, vec_x, pair;
};
struct FwdList { FwdProblem p[MAX_PROBLEMS]; int count; };

// backward, first pass: by slices of the pixels, dW [d, C], r = sum_p dq [d] and, behind a norm, S1 = sum_p dy, S2 = sum_p dy x [C]
struct MomentProblem {
    const void *x, *g1, *g2, *w1, *w2, *gamma, *beta;    // rows of dq (and of W): the first d1 from g1 [B, d1, HW] (w1), the rest from g2 (w2)
    const float2 *stats;
    float *dw, *rsums;
    float2 *sums;                      // [B, nsplit, C]
    int B, C, d, d1, HW, groups, cpg, nsplit, slice, cblocks, jblocks, blocks, vec_x, vec_g;
};
struct MomentList { MomentProblem p[MAX_PROBLEMS]; int count; };

// backward, second pass: parameter gradients and the tail coefficients of dx
struct FoldProblem {
    const float *dw, *rsums;
    const float2 *sums, *stats;
    const void *gamma;
    float2 *tail;                      // (alpha, delta) per (image, group)
    void *grad_weight, *grad_weight2, *grad_bias, *grad_bias2, *grad_gamma, *grad_beta;
    int B, C, d, d1, HW, nsplit, groups, cpg, wblocks, blocks;
};
struct FoldList { FoldProblem p[MAX_PROBLEMS]; int count; };

// backward, third pass: dx = rstd gamma_c sum_j W_jc dq_j + alpha_g x + delta_g + add
struct DxProblem {
    const void *x, *g1, *g2, *w1, *w2, *gamma, *add;
    const float2 *stats, *tail;        // nullptr: no norm
    void *out;
    int B, C, d, d1, HW, groups, cpg, mblocks, pblocks, blocks, vec_g, pair;
};
struct DxList { DxProblem p[MAX_PROBLEMS]; int count; };

}  // namespace pmm
}  // namespace sapa
