// FP64 KRP draw with certified fixed-point descents (descent_fx.cuh): per
// sample the steps of krp_draw_kernel<., double> (krp_draw.cu), the decisions
// of both descents and of the leaf scan from fixed-point and FP32 forms where
// those are certain, from the FP64 code of descent.cuh where they are not.
// The FP64 work left per sample is h o W[u], the update of h and the weight.
//
// Measured (one GB300; FP64 forms before, this kernel with its mass table now):
// N = 3, I = 2^22, R = 32, J = 50,000, one mode excluded 6.25 -> 1.66 ms; N = 4, I =
// 1000, R = 8, J = 10,000 with copies to the host 0.93 -> 0.19 ms.  It is bound by
// issue (60% of the slots at I = 2^20, R = 32; the integer pipe, which cuts the
// FP64 values, 49% of its peak) and the latency of the node reads.
//
// One warp per sample up to R = 64 (at R = 32 a query's outer product takes
// 4.2 KB of shared memory; 32 warps of 64 registers per SM measured 3% faster
// than 24 of 80); above, a team of four warps shares one sample, since a query of
// R = 100 takes 40 KB and one warp per sample would leave five warps on an SM.
#include <algorithm>

#include "descent_fx.cuh"

namespace ftl {

template <int RMAX>
struct FxShape {
    static constexpr int TW = RMAX <= 64 ? 1 : 4;          // warps per sample
    static constexpr int TEAMS = RMAX <= 64 ? 4 : 1;       // samples per block
    static constexpr int THREADS = 32 * TW * TEAMS;
    static constexpr int MINB = RMAX <= 32 ? 8 : (RMAX <= 64 ? 3 : 4);  // blocks per SM
};

// Block header: exponents of the roots, a redo's result, then the pair table.
constexpr int kFxHead = 2 * FTL_MAX_MODES * (int)sizeof(int) + 16;
__host__ __device__ inline size_t fx_head(int R) {
    return kFxHead + ((size_t)(node_stride(R, 8) / 2) * sizeof(uint16_t) + 15) / 16 * 16;
}

// Shared memory of one team, and where its parts lie.
template <int RMAX>
struct FxSmem {
    size_t slot, xd, xs, qrow, red, team;
    __host__ __device__ explicit FxSmem(int R) {
        constexpr int ROW = 32 * FxShape<RMAX>::TW;
        const int nvec = node_stride(R, 8) / 2;
        size_t o = 0;
        slot = o;
        o += (size_t)((nvec + ROW - 1) / ROW * ROW) * sizeof(float4);
        xd = o;
        o += RMAX * sizeof(double);
        xs = o;
        o += RMAX * sizeof(float2);
        qrow = o;
        o += RMAX * sizeof(float);
        red = o;
        o += 2 * FxShape<RMAX>::TW * sizeof(int2);
        team = (o + 15) / 16 * 16;
    }
};

// xx of the FP64 form into the team's slot (QForm<., double>::setup's values).
__device__ __forceinline__ void fx_fill64(double *s, const double *x, const uint16_t *pairs, int R, int P, int S,
                                          int lane) {
    for (int v = lane; 2 * v < S; v += 32) {
        const unsigned pr = pairs[v];
        int a = (int)(pr >> 8), b = (int)(pr & 0xffu);
        double o[2] = {0.0, 0.0};
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            if (2 * v + w < P) {
                o[w] = x[a] * x[b];
                if (a != b) o[w] += o[w];
            }
            if (++b == R) b = ++a;
        }
        *reinterpret_cast<double2 *>(s + 2 * v) = make_double2(o[0], o[1]);
    }
    __syncwarp();
}

// The FP64 descent (and leaf scan, with_rows) of one sample by one warp; the
// staged query is in xd, the slot is overwritten.  Returns the row with_rows,
// else the leaf index.
template <int RMAX>
__device__ __noinline__ int64_t fx_redo(const DrawParams &p, const double *G, const DGeom &g, const double *U,
                                        double *slot, const double *xd, const uint16_t *pairs, double u,
                                        bool with_rows, int lane) {
    QForm<RMAX, double> qf;
    qf.P = p.P;
    qf.S = p.S;
    qf.s = slot;
    fx_fill64(slot, xd, pairs, p.R, p.P, p.S, lane);
    double frac;
    const int64_t c = descend<RMAX>(G, p.S, g, u, qf, lane, frac);
    if (!with_rows || g.F <= 1) return leaf_index(g, c);
    bool empty;
    return leaf_scan<RMAX, double, double>(U, p.R, g, c, frac, lane_query<RMAX, double>(xd, p.R, lane), lane, empty);
}

// The block's pair table and root exponents (eg: [eigen trees, Gram trees][N]),
// and this thread's team.
template <int RMAX>
__device__ __forceinline__ void fx_setup(const DrawParams &p, unsigned char *smem, FxTeam<RMAX, FxShape<RMAX>::TW> &tm) {
    using Sh = FxShape<RMAX>;
    constexpr int TW = Sh::TW, TEAMS = Sh::TEAMS;
    const int R = p.R, N = p.N, lane = threadIdx.x & 31;
    const size_t eig_stride = (size_t)(2 * R - 1) * p.S;
    int *eg = (int *)smem;
    const FxSmem<RMAX> lay(R);
    uint16_t *pairs = (uint16_t *)(smem + kFxHead);
    unsigned char *base = smem + fx_head(R) + (threadIdx.x / (32 * TW)) * lay.team;
    tm.slot = (float4 *)(base + lay.slot);
    tm.xd = (double *)(base + lay.xd);
    tm.xs = (float2 *)(base + lay.xs);
    tm.qrow = (float *)(base + lay.qrow);
    tm.red = (int2 *)(base + lay.red);
    tm.pairs = pairs;
    tm.tid = threadIdx.x % (32 * TW);
    tm.nvec = p.S / 2;
    tm.fr = tm.nvec / (32 * TW);
    tm.flip = 0;
    for (int v = threadIdx.x; v < tm.nvec; v += Sh::THREADS) {
        int a, b;
        pair_of(min(2 * v, p.P - 1), R, a, b);
        pairs[v] = (uint16_t)((a << 8) | b);
    }
    for (int k = threadIdx.x >> 5; k < 2 * N; k += TW * TEAMS) {
        const int mode = k % N;
        unsigned e = 0;
        if ((uint32_t)mode != p.j) {
            const double *G = k < N ? (const double *)p.eig_G + mode * eig_stride : (const double *)p.gram_G[mode];
            for (int a = lane; a < R; a += 32)
                e = max(e, ((unsigned)__double2hiint(G[packed_row_offset(a, R)]) >> 20) & 0x7ffu);
        }
        e = __reduce_max_sync(0xffffffffu, e);
        if (lane == 0) eg[k] = (int)e;
    }
    __syncthreads();
}

// Mass table of the first sampled mode (draw_params.cuh): a team stages one
// query -- component u's W[u], or h = 1 for the eigen tree -- and evaluates a
// run of nodes with it.  A query or tree outside the scaling's range gives
// zeros, which the descents leave to the FP64 code.
constexpr int kFxTabRun = 16;

static __host__ __device__ int64_t fx_table_items(const DrawParams &p) {
    return (p.R + kFxTabRun - 1) / kFxTabRun +
           (int64_t)(((1 << p.tab_levels) + kFxTabRun - 1) / kFxTabRun) * p.R;
}

template <int RMAX, int FR>
__global__ void __launch_bounds__(FxShape<RMAX>::THREADS, FxShape<RMAX>::MINB) krp_table_fx_kernel(DrawParams p) {
    using Sh = FxShape<RMAX>;
    constexpr int TW = Sh::TW, TEAMS = Sh::TEAMS;
    constexpr int XPL = Shape<RMAX>::XPL;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    FxTeam<RMAX, TW> tm;
    fx_setup<RMAX>(p, smem_raw, tm);
    const int *eg = (const int *)smem_raw;
    const int R = p.R, lane = threadIdx.x & 31, k = p.tab_mode;
    const int runs = ((1 << p.tab_levels) + kFxTabRun - 1) / kFxTabRun, eruns = (R + kFxTabRun - 1) / kFxTabRun;
    const int64_t items = fx_table_items(p);
    for (int64_t it = (int64_t)blockIdx.x * TEAMS + threadIdx.x / (32 * TW); it < items;
         it += (int64_t)gridDim.x * TEAMS) {
        const bool gram = it >= eruns;
        const int u = gram ? (int)((it - eruns) / runs) : 0;
        const int t0 = (gram ? (int)((it - eruns) % runs) : (int)it) * kFxTabRun;
        const int t1 = min(gram ? 1 << p.tab_levels : R, t0 + kFxTabRun);
        double x[XPL];
#pragma unroll
        for (int q = 0; q < XPL; ++q) {
            const int col = lane + 32 * q;
            x[q] = 0.0;
            if (col < R) x[q] = gram ? p.M[(size_t)p.offset[k] * R * R + (size_t)u * R + col] : 1.0;
        }
        FxScale sc;
        const bool ok = fx_stage(tm, x, R, eg[(gram ? p.N : 0) + k], sc);
        const double *G = gram ? (const double *)p.gram_G[k] : (const double *)p.eig_G + (size_t)k * (2 * R - 1) * p.S;
        int64_t *tab = (int64_t *)p.table + (gram ? kTabEig + (size_t)u * kTabNodes : 0);
        for (int t = t0; t < t1; ++t) {
            int64_t m = 0;
            if (ok) m = fx_eval<RMAX, TW, FR>(tm, G + (size_t)(t == 0 ? 0 : 2 * t - 1) * p.S, sc);
            if (tm.tid == 0) tab[t] = m;
        }
    }
}

template <int RMAX, int FR>
__global__ void __launch_bounds__(FxShape<RMAX>::THREADS, FxShape<RMAX>::MINB) krp_draw_fx_kernel(DrawParams p) {
    using Sh = FxShape<RMAX>;
    constexpr int TW = Sh::TW, TEAMS = Sh::TEAMS;
    constexpr int XPL = Shape<RMAX>::XPL;
    using Team = FxTeam<RMAX, TW>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int R = p.R, N = p.N, lane = threadIdx.x & 31;
    const size_t RR = (size_t)R * R;
    const size_t eig_stride = (size_t)(2 * R - 1) * p.S;
    const int *eg = (const int *)smem_raw;
    int64_t *answer = (int64_t *)(smem_raw + 2 * FTL_MAX_MODES * sizeof(int));  // TW > 1: a redo's result
    Team tm;
    fx_setup<RMAX>(p, smem_raw, tm);

    const int64_t teams = (int64_t)gridDim.x * TEAMS;
#pragma unroll 1
    for (int64_t i = (int64_t)blockIdx.x * TEAMS + threadIdx.x / (32 * TW); i < p.J; i += teams) {
        // lane l < 2N holds uniform l (phase l / N, mode l % N) as 53 bits
        uint64_t D = 0;
        bool dok = true;
        if (lane < 2 * N) {
            const int64_t idx = (int64_t)lane * p.J + i;
            if (p.draws) {
                const double u = p.draws[idx];
                dok = u >= 0.0 && u < 1.0;
                if (dok) D = (uint64_t)(u * 9007199254740992.0);
            } else {
                D = philox_bits53(p.seed, p.ctr + (uint64_t)idx);
            }
        }
        const unsigned dmask = __ballot_sync(0xffffffffu, dok);
        double h[XPL];
#pragma unroll
        for (int q = 0; q < XPL; ++q) h[q] = 1.0;
#pragma unroll 1
        for (int k = 0; k < N; ++k) {
            if ((uint32_t)k == p.j) continue;
            double x[XPL];
#pragma unroll
            for (int q = 0; q < XPL; ++q) x[q] = lane + 32 * q < R ? h[q] : 0.0;
            int64_t comp = 0;  // eigen component
#pragma unroll 1
            for (int phase = 0; phase < 2; ++phase) {
                const double *G = phase == 0 ? (const double *)p.eig_G + k * eig_stride : (const double *)p.gram_G[k];
                const DGeom &g = phase == 0 ? p.eig : p.gram[k];
                const int l = phase * N + k;
                const uint64_t Dk = __shfl_sync(0xffffffffu, D, l);
                FxScale sc;
                FxLeaf lf;
                // the first sampled mode: eigen component and upper Gram levels from the mass table
                const bool tabled = p.table != nullptr && k == p.tab_mode;
                const int64_t *tab = nullptr;
                int tab_levels = -1;
                if (tabled) {
                    tab = (const int64_t *)p.table + (phase == 0 ? 0 : kTabEig + comp * kTabNodes);
                    tab_levels = phase == 0 ? kTabLevels : p.tab_levels;
                }
                const bool staged = !tabled || phase == 1;
                bool ok = (!staged || fx_stage(tm, x, R, eg[l], sc)) && ((dmask >> l) & 1u);
                int64_t t = 0;
                if (ok) {
                    if (is_leaf(g, 0)) {  // the leaf fraction is the draw
                        lf.c = 0;
                        lf.t = (int64_t)Dk;
                        lf.m = (int64_t)1 << 53;
                        lf.tol = lf.mtol = 1;
                    } else {
                        ok = fx_descend<RMAX, TW, FR>(tm, G, p.S, g, Dk, sc, lf, tab, tab_levels);
                    }
                }
                if (ok) {
                    if (phase == 1 && g.F > 1)
                        ok = fx_leaf_scan(tm, p.U[k], R, g, lf, eg[l], t);
                    else
                        t = leaf_index(g, (int64_t)lf.c);
                }
                if (!ok) {
                    const double u = get_draw(p, (int64_t)l * p.J + i);
                    if (!staged) fx_stage(tm, x, R, eg[l], sc);
                    Team::sync();
                    if (TW == 1 || tm.tid < 32) {
                        t = fx_redo<RMAX>(p, G, g, p.U[k], (double *)tm.slot, tm.xd, tm.pairs, u, phase == 1, lane);
                        if (TW > 1 && lane == 0) *answer = t;
                    }
                    Team::sync();
                    if (TW > 1) t = *answer;
                    Team::sync();
                }
                if (phase == 0) {
                    comp = t;
                    const double *Wr = p.M + (size_t)p.offset[k] * RR + (size_t)t * R;
#pragma unroll
                    for (int q = 0; q < XPL; ++q) {
                        const int col = lane + 32 * q;
                        x[q] = col < R ? h[q] * Wr[col] : 0.0;
                    }
                } else {
                    const double *Ur = p.U[k] + t * R;
#pragma unroll
                    for (int q = 0; q < XPL; ++q) {
                        const int col = lane + 32 * q;
                        if (col < R) h[q] *= Ur[col];
                    }
                    if (tm.tid == 0) p.samples[(int64_t)k * p.J + i] = (uint64_t)t;
                }
            }
        }
        if (TW == 1 || tm.tid < 32) {
            if (p.weights) {
                __syncwarp();
#pragma unroll
                for (int q = 0; q < XPL; ++q)
                    if (lane + 32 * q < R) tm.xd[lane + 32 * q] = h[q];
                __syncwarp();
                QForm<RMAX, double> qf;
                qf.P = p.P;
                qf.S = p.S;
                qf.s = (double *)tm.slot;
                fx_fill64(qf.s, tm.xd, tm.pairs, R, p.P, p.S, lane);
                const double lev = qf.eval(p.M + cm_pinv64_offset(N, R), lane);
                if (lane == 0) p.weights[i] = (double)R / (lev * (double)p.J);
            }
            if (p.h) {
#pragma unroll
                for (int q = 0; q < XPL; ++q)
                    if (lane + 32 * q < R) p.h[i * R + lane + 32 * q] = h[q];
            }
        }
        Team::sync();
    }
}

template <int RMAX, int FR>
static int launch_fx(const DrawParams &p, cudaStream_t st) {
    using Sh = FxShape<RMAX>;
    const auto kernel = krp_draw_fx_kernel<RMAX, FR>;
    const size_t smem = fx_head(p.R) + Sh::TEAMS * FxSmem<RMAX>(p.R).team;
    int rc = ensure_smem((const void *)kernel, smem, "krp_draw_fx_kernel");
    if (rc) return rc;
    // one wave of resident blocks, each looping over samples
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, Sh::THREADS, smem) != cudaSuccess || occ < 1)
        occ = 1;
    if (p.table) {
        const auto table = krp_table_fx_kernel<RMAX, FR>;
        rc = ensure_smem((const void *)table, smem, "krp_table_fx_kernel");
        if (rc) return rc;
        const int64_t tneed = (fx_table_items(p) + Sh::TEAMS - 1) / Sh::TEAMS;
        table<<<(int)std::min<int64_t>(tneed, (int64_t)num_sms() * occ), Sh::THREADS, smem, st>>>(p);
        rc = check_launch("krp_table_fx_kernel");
        if (rc) return rc;
    }
    const int64_t need = (p.J + Sh::TEAMS - 1) / Sh::TEAMS;
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>(need, (int64_t)num_sms() * occ));
    kernel<<<blocks, Sh::THREADS, smem, st>>>(p);
    return check_launch("krp_draw_fx_kernel");
}

int launch_draw_fx(const DrawParams &p, cudaStream_t st) {
    if (p.R > 64) return launch_fx<128, -1>(p, st);
    if (p.R > 32) return launch_fx<64, -1>(p, st);
    switch (p.S / 64) {  // full rows of 32 two-entry vectors in a node
        case 0: return launch_fx<32, 0>(p, st);
        case 1: return launch_fx<32, 1>(p, st);
        case 2: return launch_fx<32, 2>(p, st);
        case 3: return launch_fx<32, 3>(p, st);
        case 4: return launch_fx<32, 4>(p, st);
        case 5: return launch_fx<32, 5>(p, st);
        case 6: return launch_fx<32, 6>(p, st);
        case 7: return launch_fx<32, 7>(p, st);
        default: return launch_fx<32, 8>(p, st);
    }
}

}  // namespace ftl
