// FP64 partition-tree descents whose forms run on the FP32 and integer pipes.
//
// GB300 retires one FP64 warp instruction per 64 cycles and SM sub-partition
// (0.5 TFMA/s on the chip), so a level evaluated in FP64 is bound by its
// 528 multiply-adds (R = 32), five shuffle-adds and the division of the
// cutoff.  A decision needs only the sign of draw * m - (mass left of the
// cutoff).  Here that quantity is formed in fixed point, with a bound on its
// error, and the decision is taken when it is larger than the bound; the
// rare rest (and every query or tree with infinities, NaN or a scale that the
// bound does not hold for, see fx_in_range) is redone by the FP64 descent of
// descent.cuh.  So the samples are the FP64 descent's.
//
// Arithmetic of a form sum_e g_e xx_e (g: node entries, xx: the weighted
// outer product of the query, both scaled by powers of two so that the
// largest diagonal entry of the root lies in [1, 2) and the largest |x| too):
//   * g = gh + gl, xx = xh + xl, pairs of FP32 values of 24 + 23 bits (gh and
//     gl are cut out of the FP64 bits with integer operations).
//   * s starts at C = 1.5 2^k, 2^(k-1) >= the sum of |g xx| of a thread's
//     entries, so every value of s has the spacing 2^(k-23): t = fma(gh, xh,
//     s), d = t - s (exact), e = fma(gh, xh, -d): s takes the product's upper
//     part exactly and c collects e + gh xl + gl xh.
//   * the thread's sum is the integer bits(s) - bits(C) (units of 2^(k-23))
//     and c rounded to units of 2^(k-42); both are added over the warp as
//     integers (redux.sync), so the total is a 64-bit integer in units of
//     2^(k-42) and the descent's t -= mL, t <= mL are exact.
// Error of a form, worst case, from a thread's two accumulators of n <= 9
// products: e: 9 2^(k-49); 18 additions into c, |c| <= i 1.1 2^(k-24) after i
// products: 74 2^(k-48); gl xh: 9 2^(k-49) + 2^(k-45); the bits cut off g and
// xx: 11 2^(k-48); together 102 2^(k-48) each, and 32 2^(k-48) for rounding c
// to the unit: 32 (204 + 40) 2^(k-48) = 122 units per warp and flush of c.
// kFxErr = 160 leaves room for the FP64 descent's own roundings (a few
// 2^(k-48)).
#pragma once

#include "descent.cuh"
#include "draw_params.cuh"

namespace ftl {

constexpr int kFxErr = 160;  // units per warp and flush
constexpr int kFxCh = 8;     // vectors (of two entries) per flush, plus the ragged last one

// Row and column of packed entry e (row-major upper triangle).
__device__ __forceinline__ void pair_of(int e, int R, int &a, int &b) {
    const float w = (float)(2 * R + 1);
    a = min(R - 1, max(0, (int)((w - sqrtf(w * w - 8.0f * (float)e)) * 0.5f)));
    while (a + 1 < R && packed_row_offset(a + 1, R) <= e) ++a;
    while (packed_row_offset(a, R) > e) --a;
    b = a + e - packed_row_offset(a, R);
}

// |v| 2^-q as h + l 2^-23, q such that FP64 exponent eb goes to FP32 exponent
// 127 (kadj = -(eb - 127) << 20): h the upper 24 bits, l the next 23.  Values
// below 2^-126 after scaling become about 2^-126, zeros and FP64 subnormals
// among them, for eb >= 127 (fx_in_range; below, kadj > 0 would lift them).
__device__ __forceinline__ void fx_split(uint32_t hi, uint32_t lo, int kadj, float &h, float &l) {
    const uint32_t sg = hi & 0x80000000u;
    const int a = __viaddmax_s32((int)(hi & 0x7fffffffu), kadj, 0x00100000);
    const uint32_t r = __funnelshift_l(lo, (uint32_t)a, 3);
    const uint32_t hs = r | sg;
    h = __uint_as_float(hs);
    l = __uint_as_float(((lo >> 6) & 0x7fffffu) | (hs & 0xff800000u)) - __uint_as_float(hs & 0xff800000u);
}

// The upper part alone.
__device__ __forceinline__ float fx_upper(uint32_t hi, uint32_t lo, int kadj) {
    const int a = __viaddmax_s32((int)(hi & 0x7fffffffu), kadj, 0x00100000);
    return __uint_as_float(__funnelshift_l(lo, (uint32_t)a, 3) | (hi & 0x80000000u));
}

// Scale of one descent: the root's exponent, the accumulators' start and the
// unit.
struct FxScale {
    int kadj;      // node exponent adjustment (fx_split)
    uint32_t cb;   // bits of C
    float lscale;  // 2^(42 - k)
};

// A team of TW warps descends one sample; everything it shares.
template <int RMAX, int TW>
struct FxTeam {
    float4 *slot;  // per vector (xh0, xl0, xh1, xl1), padded to whole rows of the team
    double *xd;    // the query in FP64
    float2 *xs;    // the scaled query as (upper, lower) FP32 parts
    float *qrow;   // leaf scan: squared forms by row
    int2 *red;     // TW > 1: two sets of per-warp partial sums
    const uint16_t *pairs;  // per vector: row and column (a << 8 | b) of its first entry
    int tid;       // thread of the team
    int nvec, fr;  // vectors per node; rows of 32 TW vectors that are full
    int flip;

    static __device__ __forceinline__ void sync() {
        if constexpr (TW == 1) __syncwarp();
        else __syncthreads();
    }
};

__device__ __forceinline__ void fx_term(uint32_t hi, uint32_t lo, float xh, float xl, int kadj, float &s, float &c,
                                        float &d) {
    float gh, gl;
    fx_split(hi, lo, kadj, gh, gl);
    const float t = fmaf(gh, xh, s);
    const float up = t - s;
    s = t;
    c += fmaf(gh, xh, -up);
    c = fmaf(gh, xl, c);
    d = fmaf(gl, xh, d);
}

// The form of the staged query against a node, in units of 2^(k-42).  FR >= 0:
// the number of full rows, known at compile time (R <= 32; branch-free).
template <int RMAX, int TW, int FR>
__device__ __forceinline__ int64_t fx_eval(FxTeam<RMAX, TW> &tm, const double *__restrict__ node, const FxScale &sc) {
    constexpr int ROW = 32 * TW;
    const uint4 *nv = reinterpret_cast<const uint4 *>(node) + tm.tid;
    const float4 *xv = tm.slot + tm.tid;
    const int fr = FR >= 0 ? FR : tm.fr;
    int hi = 0, lo = 0;
    int u0 = 0;
#pragma unroll 1
    do {
        uint4 g[kFxCh], gt = make_uint4(0, 0, 0, 0);
        const bool last = u0 + kFxCh >= fr, whole = u0 + kFxCh <= fr;
        if (FR < 0 && whole) {
#pragma unroll
            for (int u = 0; u < kFxCh; ++u) g[u] = __ldg(nv + (u0 + u) * ROW);
        } else {
#pragma unroll
            for (int u = 0; u < kFxCh; ++u)
                if (u0 + u < fr) g[u] = __ldg(nv + (u0 + u) * ROW);
        }
        if (last && tm.tid + fr * ROW < tm.nvec) gt = __ldg(nv + fr * ROW);
        float s0 = __uint_as_float(sc.cb), s1 = s0, c0 = 0.0f, c1 = 0.0f, d0 = 0.0f, d1 = 0.0f;
        auto term = [&](const uint4 &v, int u) {
            const float4 x = xv[u * ROW];
            fx_term(v.y, v.x, x.x, x.y, sc.kadj, s0, c0, d0);
            fx_term(v.w, v.z, x.z, x.w, sc.kadj, s1, c1, d1);
        };
        if (FR < 0 && whole) {
#pragma unroll
            for (int u = 0; u < kFxCh; ++u) term(g[u], u0 + u);
        } else {
#pragma unroll
            for (int u = 0; u < kFxCh; ++u)
                if (u0 + u < fr) term(g[u], u0 + u);
        }
        if (last && fr * ROW < tm.nvec) term(gt, fr);  // xx is zero past the node
        hi += (int)(__float_as_uint(s0) - sc.cb) + (int)(__float_as_uint(s1) - sc.cb);
        lo += __float2int_rn(fmaf(d0 + d1, 1.1920928955078125e-07f, c0 + c1) * sc.lscale);
        u0 += kFxCh;
    } while (FR < 0 && u0 < fr);
    hi = __reduce_add_sync(0xffffffffu, hi);
    lo = __reduce_add_sync(0xffffffffu, lo);
    if constexpr (TW == 1) {
        return ((int64_t)hi << 19) + lo;
    } else {
        int2 *r = tm.red + TW * tm.flip;
        tm.flip ^= 1;
        if ((tm.tid & 31) == 0) r[tm.tid >> 5] = make_int2(hi, lo);
        __syncthreads();
        int64_t m = 0;
#pragma unroll
        for (int w = 0; w < TW; ++w) m += ((int64_t)r[w].x << 19) + r[w].y;
        return m;
    }
}

// Flushes of a form (its error is kFxErr TW times this).
template <int RMAX, int TW>
__device__ __forceinline__ int fx_flushes(const FxTeam<RMAX, TW> &tm) {
    return max(1, (tm.fr + kFxCh - 1) / kFxCh);
}

// (2 - [a == b]) x_a x_b as an upper and a lower FP32 part.
__device__ __forceinline__ void fx_product(const float2 *xs, int a, int b, float &ph, float &pl) {
    const float2 xa = xs[a], xb = xs[b];
    const float f = a == b ? 1.0f : 2.0f;
    const float ah = f * xa.x, al = f * xa.y;
    const float p = ah * xb.x;
    const float q = fmaf(al, xb.x, fmaf(ah, xb.y, fmaf(ah, xb.x, -p)));
    ph = p + q;
    pl = q - (ph - p);
}

// Whether queries whose largest FP64 exponent is emax may be scaled against
// trees whose root's largest diagonal exponent is eg: both exponents are at
// least 127 (fx_split), and the products x_a x_b and g x_a x_b of the largest
// entries keep FP64's full precision, so that the FP64 forms are rounded sums
// as the error bound takes them to be and neither lose bits in subnormals nor
// overflow.
__device__ __forceinline__ bool fx_in_range(int emax, int eg) {
    const int x = emax - 1023, m = eg - 1023 + 2 * x;
    return eg >= 127 && eg < 2046 && x >= -448 && x <= 480 && m >= -896 && m <= 960;
}

// Stage query x (FP64, XPL entries per lane, every warp of the team holds it)
// for fx_eval against trees whose root's largest diagonal exponent is eg.
// Returns false (uniformly) when the scaling does not hold.
template <int RMAX, int TW>
__device__ __forceinline__ bool fx_stage(FxTeam<RMAX, TW> &tm, const double (&x)[Shape<RMAX>::XPL], int R, int eg,
                                         FxScale &sc) {
    constexpr int XPL = Shape<RMAX>::XPL;
    constexpr int ROW = 32 * TW;
    const int lane = tm.tid & 31;
    unsigned emax = 0;
#pragma unroll
    for (int q = 0; q < XPL; ++q) emax = max(emax, ((unsigned)__double2hiint(x[q]) >> 20) & 0x7ffu);
    emax = __reduce_max_sync(0xffffffffu, emax);
    FxTeam<RMAX, TW>::sync();
    if (tm.tid < 32) {
        const int xadj = -((int)emax - 127) * (1 << 20);
#pragma unroll
        for (int q = 0; q < XPL; ++q) {
            const int col = lane + 32 * q;
            if (col < R) {
                float h, l;
                fx_split((uint32_t)__double2hiint(x[q]), (uint32_t)__double2loint(x[q]), xadj, h, l);
                tm.xs[col] = make_float2(h, l * 1.1920928955078125e-07f);
                tm.xd[col] = x[q];
            }
        }
    }
    FxTeam<RMAX, TW>::sync();
    if (!fx_in_range((int)emax, eg)) return false;
    const int P = packed_size(R);
    float bmax = 0.0f, b0 = 0.0f, b1 = 0.0f;
    for (int u = 0; u * ROW < tm.nvec; ++u) {
        const int v = u * ROW + tm.tid;
        float4 o = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (2 * v < P) {
            const unsigned pr = tm.pairs[v];
            int a = (int)(pr >> 8), b = (int)(pr & 0xffu);
            fx_product(tm.xs, a, b, o.x, o.y);
            if (++b == R) b = ++a;
            if (2 * v + 1 < P) fx_product(tm.xs, a, b, o.z, o.w);
        }
        tm.slot[v] = o;
        // sums of |xx| per accumulator and flush (the ragged row joins the last)
        if (u % kFxCh == 0 && u < tm.fr) b0 = b1 = 0.0f;
        b0 += fabsf(o.x);
        b1 += fabsf(o.z);
        bmax = fmaxf(bmax, fmaxf(b0, b1));
    }
    unsigned bb = __reduce_max_sync(0xffffffffu, __float_as_uint(bmax));
    if constexpr (TW > 1) {
        int2 *r = tm.red + TW * tm.flip;
        tm.flip ^= 1;
        if (lane == 0) r[tm.tid >> 5].x = (int)bb;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < TW; ++w) bb = max(bb, (unsigned)r[w].x);
    } else {
        __syncwarp();
    }
    const int ex = (int)(__float_as_uint(__uint_as_float(bb) * 1.001f) >> 23);
    sc.kadj = -(eg - 127) * (1 << 20);
    sc.cb = ((uint32_t)(ex + 3) << 23) | 0x400000u;
    sc.lscale = __uint_as_float((uint32_t)(293 - ex) << 23);
    return true;
}

// Outcome of a certified descent: the leaf, and the draw's offset in it.
struct FxLeaf {
    uint32_t c;
    int64_t t, m;       // offset and mass, in units
    int64_t tol, mtol;  // their error bounds
};

// The descent of descent.cuh's FP64 `descend` for uniform D 2^-53; false when
// a decision is closer than the error bound.  The forms of the root and of the
// first tab_levels levels come from a mass table (tab_levels = -1: none).
template <int RMAX, int TW, int FR>
__device__ __forceinline__ bool fx_descend(FxTeam<RMAX, TW> &tm, const double *__restrict__ G, int S, const DGeom &g,
                                           uint64_t D, const FxScale &sc, FxLeaf &out, const int64_t *tab,
                                           int tab_levels) {
    const int64_t E = (int64_t)kFxErr * TW * fx_flushes(tm);
    const uint32_t ncount = (uint32_t)g.node_count;
    const int lf = (int)g.lfill_level;
    uint32_t c = 0;
    int64_t t = 0, m = 0, tol = 2 * E + 4, mtol = E;
    const double *node = G;
#pragma unroll 1
    for (int lvl = -1;; ++lvl) {
        int64_t f;
        if (lvl < tab_levels) f = __ldg((const long long *)tab + (lvl < 0 ? 0 : 1 + c));
        else f = fx_eval<RMAX, TW, FR>(tm, node, sc);
        if (lvl < 0) {
            if (f <= 16 * E) return false;
            m = f;
            t = (int64_t)__umul64hi(D << 11, (uint64_t)f);
        } else {
            const int64_t d = t - f;
            if (llabs(d) <= tol) return false;
            if (d < 0) {
                c = 2 * c + 1;
                m = f;
                mtol = E;
            } else {
                c = 2 * c + 2;
                t = d;
                tol += E;
                m -= f;
                mtol += E;
            }
            if (lvl == lf) break;
        }
        if (lvl + 1 == lf && 2u * c + 1u >= ncount) break;
        node = G + (size_t)(2u * c + 1u) * (size_t)S;
    }
    out.c = c;
    out.t = t;
    out.m = m;
    out.tol = tol;
    out.mtol = mtol;
    return true;
}

// Row of leaf block c for the offset lf.t: the FP64 rule (first row r <= F - 2
// with t/m < prefix_r / total, else the last) on forms rounded to FP32, taken
// when no row boundary lies within the error bound; false otherwise.  The
// offset inside one block needs no more than FP32: a boundary is that close
// for about one sample in 10^3.
// Error: q_r = sum_a u_ra x_a is off by at most gamma A_r, A_r = sum |u_ra x_a|,
// gamma = 2^-20 (x and u cut to 24 bits, at most nine roundings of the sum;
// u is scaled by a power of two above the root of the tree's largest diagonal
// entry, so no |u| exceeds 2 and what underflows is far below the total that
// is asked for); sum_r A_r^2 <= R sum_ra (u_ra x_a)^2 = R S, so the sum of the q_r^2 is
// off by at most 2 gamma sqrt(total R S) + gamma^2 R S.
template <int RMAX, int TW>
__device__ __forceinline__ bool fx_leaf_scan(FxTeam<RMAX, TW> &tm, const double *__restrict__ U, int R, const DGeom &g,
                                             const FxLeaf &lf, int eg, int64_t &row) {
    constexpr int XPL = Shape<RMAX>::XPL, FQ = Shape<RMAX>::FQ;
    constexpr int K = 16;
    const int lane = tm.tid & 31, warp = tm.tid >> 5;
    const int F = (int)g.F;
    const int64_t row0 = leaf_index(g, (int64_t)lf.c) * g.F;
    const int rows = (int)min((int64_t)F, g.n - row0);
    float x[XPL];
#pragma unroll
    for (int q = 0; q < XPL; ++q) x[q] = lane + 32 * q < R ? tm.xs[lane + 32 * q].x : 0.0f;
    float sq = 0.0f;
    const int uadj = -((eg + 1023) / 2 + 1 - 127) * (1 << 20);
#pragma unroll 1
    for (int r0 = K * warp; r0 < F; r0 += K * TW) {
        float v[K];
#pragma unroll
        for (int rr = 0; rr < K; ++rr) {
            v[rr] = 0.0f;
            if (r0 + rr < rows) {
                const uint2 *u = reinterpret_cast<const uint2 *>(U + (row0 + r0 + rr) * (int64_t)R);
#pragma unroll
                for (int q = 0; q < XPL; ++q)
                    if (lane + 32 * q < R) {
                        const uint2 w = __ldg(u + lane + 32 * q);
                        const float p = fx_upper(w.y, w.x, uadj) * x[q];
                        v[rr] += p;
                        sq = fmaf(p, p, sq);
                    }
            }
        }
        const float f = transpose_reduce<K, float>(v, lane);  // row r0 + lane / 2
        if ((lane & 1) == 0) tm.qrow[r0 + (lane >> 1)] = f * f;
    }
    sq = warp_sum(sq);
    float stot = sq;
    if constexpr (TW > 1) {
        int2 *r = tm.red + TW * tm.flip;
        tm.flip ^= 1;
        if (lane == 0) r[warp].x = __float_as_int(sq);
        __syncthreads();
        stot = 0.0f;
#pragma unroll
        for (int w = 0; w < TW; ++w) stot += __int_as_float(r[w].x);
    } else {
        __syncwarp();
    }
    float incl[FQ], tot = 0.0f;
#pragma unroll
    for (int q = 0; q < FQ; ++q) {
        float v = lane + 32 * q < F ? tm.qrow[lane + 32 * q] : 0.0f;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float up = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += up;
        }
        incl[q] = v + tot;
        tot += __shfl_sync(0xffffffffu, v, 31);
    }
    const float m = (float)lf.m, f = (float)lf.t / m;
    const float df = ((float)lf.tol + f * (float)lf.mtol) / m * 1.01f;
    const float rs = (float)R * stot * 1.01f;
    const float dq = 2.1f * 9.5367431640625e-07f * sqrtf(tot * rs) + 9.5367431640625e-07f * 9.5367431640625e-07f * rs;
    const float thr = f * tot, err = df * tot + 2.1f * dq + 1.9073486328125e-06f * tot;
    bool ok = tot > 1e-30f && tot < 1e30f && err < tot && m > 0.0f;
    int res = F - 1;
#pragma unroll
    for (int q = FQ - 1; q >= 0; --q) {
        const int r = lane + 32 * q;
        const unsigned bal = __ballot_sync(0xffffffffu, r <= F - 2 && thr < incl[q]);
        if (bal) res = 32 * q + (__ffs(bal) - 1);
        ok = ok && !(r <= F - 2 && !(fabsf(thr - incl[q]) > err));
    }
    row = row0 + min(res, rows - 1);
    return __all_sync(0xffffffffu, ok);
}

}  // namespace ftl
