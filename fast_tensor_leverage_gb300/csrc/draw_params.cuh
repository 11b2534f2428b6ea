// Parameters of one draw's descent kernels and the source of its uniforms.
#pragma once

#include "ftl_common.cuh"

namespace ftl {

struct DrawParams {
    int N, R, P, S;
    uint32_t j;
    int64_t J;
    DGeom gram[FTL_MAX_MODES];
    DGeom eig;
    const double *U[FTL_MAX_MODES];
    const float *U32[FTL_MAX_MODES];  // FP32 copies of U for the leaf scans (S32 kernels)
    const void *gram_G[FTL_MAX_MODES];
    const void *eig_G;
    const double *M;
    const float *pinv32;
    int offset[FTL_MAX_MODES];
    uint64_t *samples;
    double *h;
    double *weights;
    const double *draws;
    uint64_t seed, ctr;
};

__device__ __forceinline__ double get_draw(const DrawParams &p, int64_t idx) {
    return p.draws ? p.draws[idx] : philox_uniform(p.seed, p.ctr + (uint64_t)idx);
}

}  // namespace ftl
