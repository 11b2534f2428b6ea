// Parameters of one draw's descent kernels and the source of its uniforms.
#pragma once

#include "ftl_common.cuh"

namespace ftl {

// Mass table of a draw's first sampled mode.  There h = 1, so every sample
// asks the same question of the eigen tree and one of R questions (W[u]) of
// the top of the Gram tree; the answers are the forms the descent would
// evaluate, so a descent that reads them takes the same decisions.  Entries
// (FP32 trees: FP32 forms; FP64 trees: int64 forms in units of descent_fx.cuh):
// [0, kTabEig): the eigen tree with query h = 1; then kTabNodes per component
// u: the Gram tree with query W[u].  Entry 0 of either: the root; entry 1 + c:
// the left child of node c.
constexpr int kTabEig = 256;          // root and up to 127 left children
constexpr int kTabLevels = 12;        // Gram-tree levels at most
constexpr int kTabNodes = 1 << kTabLevels;
constexpr int64_t kTabMinJ = 16384;

inline size_t table_bytes(int R, int esize) { return (kTabEig + (size_t)R * kTabNodes) * esize; }

// Gram-tree levels worth tabulating for J samples: L levels cost R 2^L forms
// and save J L, so a level is added while it costs at most half of what it
// saves.  0: no table (a tree of few levels, or few samples: below three waves
// of resident warps a draw takes as long as its last wave, and the table's own
// launch was 8 us on top of 200 at N = 4, I = 1000, R = 8, J = 10,000).  FP64, N = 3, I =
// 2^22, R = 32, J = 50,000, one mode excluded (10 levels): 2.09 -> 1.77 ms;
// FP32, N = 4, R = 64, J = 32,768 (8 levels): 3.83 -> 3.70 ms.
inline int table_levels(const DGeom &g, int R, int64_t J) {
    int L = 0;
    if (J < kTabMinJ) return 0;
    while (L < kTabLevels && L < (int)g.lfill_level && (int64_t)R << (L + 1) <= J) ++L;
    return L >= 3 ? L : 0;
}

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
    void *table;   // null: none
    int tab_mode;  // the first sampled mode
    int tab_levels;
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
