// Dense symmetric eigensolver and Cholesky factorisation for one CTA,
// R x R matrices in shared (or global scratch) memory.  Used by computeM and
// by the ALS pseudo-inverse.
//
// jacobi_eigen32 (FP32) and jacobi64 (FP64): cyclic parallel-order (round-robin) two-sided Jacobi; each
// round rotates R/2 disjoint pairs (p, q) with the classical rotation that
// zeroes a_pq (tau = (a_qq - a_pp) / (2 a_pq), t = sign(tau) / (|tau| +
// sqrt(1 + tau^2)), c = 1 / sqrt(1 + t^2), s = t c), skipping pairs with
// |a_pq| <= eps sqrt(|a_pp a_qq|) (Demmel and Veselic's relative criterion);
// stops after a sweep without rotations (at most 40 sweeps).
#pragma once

#include "ftl_common.cuh"

// Stopping rule of the warp Jacobi: a pair is rotated while |a_p . a_q| >
// FTL_CM_JACOBI_TOL 2^-24 |a_p| |a_q|.
#ifndef FTL_CM_JACOBI_TOL
#define FTL_CM_JACOBI_TOL 1.0f
#endif

namespace ftl {

// In-place Jacobi on A (R x R, symmetric, row-major, FP32); V receives the
// eigenvectors as columns.  All threads of the block must call it.  (FP64:
// jacobi64 below.)
__device__ inline void jacobi_eigen32(float *A, float *V, int R, float *csbuf, int *pqbuf, int *flag) {
    using T = float;
    const int tid = threadIdx.x, nth = blockDim.x;
    const int n = R + (R & 1);
    const int half = n / 2;
    const T eps = 5.9604645e-08f;
    for (int e = tid; e < R * R; e += nth) V[e] = (e / R == e % R) ? T(1) : T(0);
    __syncthreads();
    for (int sweep = 0; sweep < 40; ++sweep) {
        if (tid == 0) *flag = 0;
        __syncthreads();
        for (int round = 0; round < n - 1; ++round) {
            if (tid < half) {
                int p, q;
                if (tid == 0) {
                    p = round;
                    q = n - 1;
                } else {
                    p = (round + tid) % (n - 1);
                    q = (round - tid + (n - 1)) % (n - 1);
                }
                if (p > q) {
                    int t = p;
                    p = q;
                    q = t;
                }
                T c = T(1), s = T(0);
                if (q < R) {
                    T apq = A[p * R + q];
                    T app = A[p * R + p];
                    T aqq = A[q * R + q];
                    if (apq != T(0) && fabs(apq) > eps * sqrt(fabs(app * aqq))) {
                        T theta = (aqq - app) / (T(2) * apq);
                        T t;
                        if (fabs(theta) > T(1e18))
                            t = T(0.5) / theta;
                        else
                            t = (theta >= T(0) ? T(1) : T(-1)) / (fabs(theta) + sqrt(T(1) + theta * theta));
                        c = T(1) / sqrt(T(1) + t * t);
                        s = t * c;
                        *flag = 1;
                    }
                }
                csbuf[2 * tid] = c;
                csbuf[2 * tid + 1] = s;
                pqbuf[2 * tid] = p;
                pqbuf[2 * tid + 1] = q;
            }
            __syncthreads();
            // A <- J^T A J and V <- V J in one pass: every entry of A lies in
            // exactly one 2 x 2 block (row pair i, column pair k), rotated by
            // columns (A J) and then by rows (J^T A), the order of the two
            // separate passes; the rotated pairs' off-diagonal entries are
            // then exact zeros.  Indices >= R (the padding pair of odd R,
            // whose rotation is the identity) have no storage.
            const int nblk = half * half;
            for (int w = tid; w < nblk + half * R; w += nth) {
                if (w < nblk) {
                    const int i = w / half, k = w - i * half;
                    const T si = csbuf[2 * i + 1], sk = csbuf[2 * k + 1];
                    if (si == T(0) && sk == T(0)) continue;
                    const T ci = csbuf[2 * i], ck = csbuf[2 * k];
                    const int pi = pqbuf[2 * i], qi = pqbuf[2 * i + 1];
                    const int pk = pqbuf[2 * k], qk = pqbuf[2 * k + 1];
                    const bool rq = qi < R, cq = qk < R;
                    T x00 = A[pi * R + pk];
                    T x01 = cq ? A[pi * R + qk] : T(0);
                    T x10 = rq ? A[qi * R + pk] : T(0);
                    T x11 = (rq && cq) ? A[qi * R + qk] : T(0);
                    if (sk != T(0)) {
                        const T t00 = ck * x00 - sk * x01, t01 = sk * x00 + ck * x01;
                        const T t10 = ck * x10 - sk * x11, t11 = sk * x10 + ck * x11;
                        x00 = t00;
                        x01 = t01;
                        x10 = t10;
                        x11 = t11;
                    }
                    if (si != T(0)) {
                        const T u00 = ci * x00 - si * x10, u10 = si * x00 + ci * x10;
                        const T u01 = ci * x01 - si * x11, u11 = si * x01 + ci * x11;
                        x00 = u00;
                        x10 = u10;
                        x01 = u01;
                        x11 = u11;
                    }
                    if (i == k) {
                        x01 = T(0);
                        x10 = T(0);
                    }
                    A[pi * R + pk] = x00;
                    if (cq) A[pi * R + qk] = x01;
                    if (rq) A[qi * R + pk] = x10;
                    if (rq && cq) A[qi * R + qk] = x11;
                } else {
                    const int w2 = w - nblk;
                    const int k = w2 / R, r = w2 - k * R;
                    const T sk = csbuf[2 * k + 1];
                    if (sk == T(0)) continue;
                    const T ck = csbuf[2 * k];
                    const int pk = pqbuf[2 * k], qk = pqbuf[2 * k + 1];
                    const T vrp = V[r * R + pk], vrq = V[r * R + qk];
                    V[r * R + pk] = ck * vrp - sk * vrq;
                    V[r * R + qk] = sk * vrp + ck * vrq;
                }
            }
            __syncthreads();
        }
        if (*flag == 0) break;
        __syncthreads();
    }
    __syncthreads();
}

// ------------------------------------------------------------ FP64 Jacobi

// Jacobi rotation of the pair (p, q) in FP64: c, s with c^2 + s^2 = 1 to FP64
// accuracy and t = s / c the small-angle solution of t^2 + 2 theta t - 1 = 0,
// theta = (a_qq - a_pp) / (2 a_pq), to FP32 accuracy: the rotation leaves
// about 2^-23 |a_pq| of the entry, which the next sweep removes with the
// second-order rest.  Returns false (no rotation) when |a_pq| <= 2^-53
// sqrt(|a_pp a_qq|).  A division or square root on GB300's FP64 pipe is some
// ten instructions of 64 cycles each; t comes from FP32 values scaled by a
// common power of two, c from an FP32 reciprocal square root x of 1 + t^2 and
// one third-order step, c = x + x e (1/2 + 3/8 e) with e = 1 - (1 + t^2) x^2
// (the series of (1 - e)^(-1/2): 2^-22 becomes below 2^-60).  An entry below
// 2^-100 of the largest of the three can still ask for a rotation (columns 30
// decades apart and more); one of a_pp, a_qq is below 2^-94 of the other then,
// t = a_pq / (a_qq - a_pp) to FP64 accuracy and the divisor is a normal FP32.
__device__ __forceinline__ bool rotation64(double app, double aqq, double apq, double &c, double &s) {
    c = 1.0;
    s = 0.0;
    const int ep = (__double2hiint(app) >> 20) & 0x7ff, eq = (__double2hiint(aqq) >> 20) & 0x7ff,
              eo = (__double2hiint(apq) >> 20) & 0x7ff;
    const int em = max(max(ep, eq), eo);
    const int sh = max(1, min(2045, 2046 - em));
    const double sc = __hiloint2double(sh << 20, 0);  // 2^(1023 - em): the largest in [1, 2)
    const double p = app * sc, q = aqq * sc, o = apq * sc;
    if (__builtin_expect(eo > max(0, em - 480) && em < 2047, 1)) {
        if (!(o * o > 1.2325951644078309e-32 * fabs(p * q))) return false;  // 2^-106
    } else {  // the squares could underflow; infinities
        if (((__double2hiint(apq) & 0x7fffffff) | __double2loint(apq)) == 0) return false;
        if (!(fabs(apq) > 1.1102230246251565e-16 * sqrt(fabs(app * aqq)))) return false;
        if (em == 2047) {  // theta = 0
            c = s = 0.70710678118654752;
            return true;
        }
    }
    const float d = d2f_rn(q - p);
    if ((__double2hiint(o) & 0x7fffffff) < ((1023 - 100) << 20)) {
        s = o * f2d_exact(1.0f / d);
        return s != 0.0;
    }
    const float b = 2.0f * d2f_rn(o);
    const float tf = fabsf(b) / (fabsf(d) + sqrtf(fmaf(d, d, b * b)));  // theta = d / b
    const double t = f2d_exact((d < 0.0f) == (b < 0.0f) ? tf : -tf);
    const double w = fma(t, t, 1.0), x = f2d_exact(rsqrtf(fmaf(tf, tf, 1.0f)));
    const double e = fma(-w * x, x, 1.0);
    c = fma(x * e, fma(0.375, e, 0.5), x);
    s = t * c;
    return true;
}

// Storage of a matrix the Jacobi method works on: shared (or this CTA's own
// global) memory, or global memory shared by the CTAs of a cluster, which is
// read and written in L2.
struct OwnMat {
    double *p;
    __device__ __forceinline__ double ld(int e) const { return p[e]; }
    __device__ __forceinline__ void st(int e, double v) const { p[e] = v; }
};
struct ClusterMat {
    double *p;
    __device__ __forceinline__ double ld(int e) const { return __ldcg(p + e); }
    __device__ __forceinline__ void st(int e, double v) const { __stcg(p + e, v); }
};

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Pair i of a round-robin round over n (even) indices, p < q.
__device__ __forceinline__ void jacobi_pair(int round, int i, int n, int &p, int &q) {
    p = i == 0 ? round : (round + i) % (n - 1);
    q = i == 0 ? n - 1 : (round - i + (n - 1)) % (n - 1);
    if (p > q) {
        const int t = p;
        p = q;
        q = t;
    }
}

// Block (i, k), k >= i, number w of the triangle of `half` pairs: row i starts
// at i half - i (i - 1) / 2.
__device__ __forceinline__ void jacobi_block(int w, int half, int &i, int &k) {
    const float f = (float)(2 * half + 1);
    i = min(half - 1, max(0, (int)((f - sqrtf(f * f - 8.0f * (float)w)) * 0.5f)));
    while (i + 1 < half && packed_row_offset(i + 1, half) <= w) ++i;
    while (packed_row_offset(i, half) > w) --i;
    k = i + w - packed_row_offset(i, half);
}

// The round's rotations of all pairs, from the matrix A.
template <class MA>
__device__ __forceinline__ void jacobi_rotations(const MA A, int R, int round, double *cs, int *pq, int *flag) {
    const int n = R + (R & 1);
    for (int i = threadIdx.x; i < n / 2; i += blockDim.x) {
        int p, q;
        jacobi_pair(round, i, n, p, q);
        double c = 1.0, s = 0.0;
        if (q < R && rotation64(A.ld(p * R + p), A.ld(q * R + q), A.ld(p * R + q), c, s)) *flag = 1;
        cs[2 * i] = c;
        cs[2 * i + 1] = s;
        pq[2 * i] = p;
        pq[2 * i + 1] = q;
    }
}

// One 2 x 2 block of the round from A into B (A and B may be the same).
template <class MA>
__device__ __forceinline__ void jacobi_rotate(const MA A, const MA B, int R, int i, int k, const double *cs,
                                              const int *pq) {
    auto at = [&](int r, int c) { return r < c ? r * R + c : c * R + r; };
    const double ci = cs[2 * i], si = cs[2 * i + 1], ck = cs[2 * k], sk = cs[2 * k + 1];
    const int pi = pq[2 * i], qi = pq[2 * i + 1], pk = pq[2 * k], qk = pq[2 * k + 1];
    const bool rq = qi < R, cq = qk < R;  // the padding index of odd R has no storage
    double x00 = A.ld(at(pi, pk));
    double x01 = cq ? A.ld(at(pi, qk)) : 0.0;
    double x10 = i == k ? x01 : (rq ? A.ld(at(qi, pk)) : 0.0);
    double x11 = (rq && cq) ? A.ld(at(qi, qk)) : 0.0;
    const double t00 = ck * x00 - sk * x01, t01 = sk * x00 + ck * x01;
    const double t10 = ck * x10 - sk * x11, t11 = sk * x10 + ck * x11;
    x00 = ci * t00 - si * t10;
    x10 = si * t00 + ci * t10;
    x01 = ci * t01 - si * t11;
    x11 = si * t01 + ci * t11;
    B.st(at(pi, pk), x00);
    if (cq) B.st(at(pi, qk), x01);
    if (rq && i != k) B.st(at(qi, pk), x10);
    if (rq && cq) B.st(at(qi, qk), x11);
}

// The two-sided Jacobi method in FP64 by one CTA: eigenvalues on the diagonal
// of A, eigenvectors in V's columns.  Only A's upper triangle is read and
// written.  Scratch: cs (R + 2 doubles), pq (R + 2 ints), flag.
__device__ inline void jacobi64(double *A, double *V, int R, double *cs, int *pq, int *flag) {
    const int tid = threadIdx.x, nth = blockDim.x;
    const int n = R + (R & 1), half = n / 2;
    const OwnMat M{A};
    for (int e = tid; e < R * R; e += nth) V[e] = (e / R == e % R) ? 1.0 : 0.0;
    if (tid == 0) *flag = 0;
    __syncthreads();
    const int ntri = half * (half + 1) / 2, nvp = half * R;
    for (int sweep = 0; sweep < 40; ++sweep) {
        for (int round = 0; round < n - 1; ++round) {
            jacobi_rotations(M, R, round, cs, pq, flag);
            __syncthreads();
            for (int w = tid; w < ntri + nvp; w += nth) {
                if (w < ntri) {
                    int i, k;
                    jacobi_block(w, half, i, k);
                    if (cs[2 * i + 1] != 0.0 || cs[2 * k + 1] != 0.0) jacobi_rotate(M, M, R, i, k, cs, pq);
                } else {
                    const int w2 = w - ntri, k = w2 / R, r = w2 - k * R;
                    const double ck = cs[2 * k], sk = cs[2 * k + 1];
                    if (sk == 0.0) continue;
                    const int pk = r * R + pq[2 * k], qk = r * R + pq[2 * k + 1];
                    const double vp = V[pk], vq = V[qk];
                    V[pk] = ck * vp - sk * vq;
                    V[qk] = sk * vp + ck * vq;
                }
            }
            __syncthreads();
        }
        const int any = *flag;
        __syncthreads();
        if (tid == 0) *flag = 0;
        if (!any) break;
        __syncthreads();
    }
    __syncthreads();
}

// The same by the nr CTAs of a cluster (this one is number rk), on two copies
// of the matrix in global memory: a round reads one and writes every block into
// the other, so that one barrier per round is enough.  The blocks are split
// over all threads; every CTA forms all the round's rotations itself from the
// same entries, so the CTAs agree on them without an exchange; a CTA keeps its
// ceil(R / nr) rows of V in shared memory (Vs) and rotates them between
// arriving at the barrier and waiting.  The wait orders what came before the
// arrivals, not these rotations of V, so a warp may form the next round's
// rotations while another still reads this round's: they are kept in two sets
// used in turn, and a set is written again two rounds later, behind the next
// round's __syncthreads, which every reader of the set has reached.  Scratch:
// cs (2 (R + 2) doubles), pq (2 (R + 2) ints), flag.  A0 holds the matrix; on
// return *eig points to the copy with the eigenvalues on its diagonal and *vec
// to the other one, which holds V.
__device__ inline void jacobi64_cluster(double *A0, double *A1, int R, double *cs, int *pq, int *flag, double *Vs,
                                        int rk, int nr, double **eig, double **vec) {
    const int tid = threadIdx.x, nth = blockDim.x;
    const int n = R + (R & 1), half = n / 2;
    const int rpc = (R + nr - 1) / nr, r0 = rk * rpc, nrows = max(0, min(R, r0 + rpc) - r0);
    for (int e = tid; e < nrows * R; e += nth) Vs[e] = (r0 + e / R == e % R) ? 1.0 : 0.0;
    if (tid == 0) *flag = 0;
    cluster_sync();
    const int ntri = half * (half + 1) / 2;
    ClusterMat src{A0}, dst{A1};
    int set = 0;
    for (int sweep = 0; sweep < 40; ++sweep) {
        for (int round = 0; round < n - 1; ++round) {
            double *c2 = cs + set * (R + 2);
            int *p2 = pq + set * (R + 2);
            set ^= 1;
            jacobi_rotations(src, R, round, c2, p2, flag);
            __syncthreads();
            for (int w = rk + nr * tid; w < ntri; w += nr * nth) {  // every CTA the same share
                int i, k;
                jacobi_block(w, half, i, k);
                jacobi_rotate(src, dst, R, i, k, c2, p2);
            }
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            for (int w = tid; w < half * nrows; w += nth) {
                const int k = w / nrows, r = w - k * nrows;
                const double ck = c2[2 * k], sk = c2[2 * k + 1];
                if (sk == 0.0) continue;
                const int pk = r * R + p2[2 * k], qk = r * R + p2[2 * k + 1];
                const double vp = Vs[pk], vq = Vs[qk];
                Vs[pk] = ck * vp - sk * vq;
                Vs[qk] = sk * vp + ck * vq;
            }
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
            const ClusterMat t = src;
            src = dst;
            dst = t;
        }
        const int any = *flag;
        __syncthreads();
        if (tid == 0) *flag = 0;
        if (!any) break;
        __syncthreads();
    }
    for (int e = tid; e < nrows * R; e += nth) dst.st(r0 * R + e, Vs[e]);
    cluster_sync();
    *eig = src.p;
    *vec = dst.p;
}

// order[r] = index of the r-th smallest eigenvalue (ties by index).
template <typename T>
__device__ void sort_ascending(const T *A, int R, int *order) {
    // A NaN on the diagonal (from a NaN input) ranks as +infinity, so the
    // ranks are always a permutation of 0..R-1 and every order[] slot is
    // written: plain < and == on NaN would give colliding ranks and leave
    // slots holding stale shared memory that callers use as indexes.
    for (int v = threadIdx.x; v < R; v += blockDim.x) {
        T lv = A[v * R + v];
        if (lv != lv) lv = T(INFINITY);
        int rank = 0;
        for (int u = 0; u < R; ++u) {
            T lu = A[u * R + u];
            if (lu != lu) lu = T(INFINITY);
            if (lu < lv || (lu == lv && u < v)) ++rank;
        }
        order[rank] = v;
    }
    __syncthreads();
}

// Eigendecomposition of a symmetric positive semidefinite R x R matrix
// (R <= 32) by one warp, in FP32: the one-sided Jacobi method of Hestenes
// ("Inversion of matrices by biorthogonalization", J. SIAM 6, 1958) on the
// columns of A.  Lane j keeps column j of A (and of V, starting at the
// identity) in registers; a round pairs the 32 columns by the round-robin
// (circle) schedule -- lane 31 meets lane r in round r, lane l meets
// (2r - l) mod 31 otherwise -- and each pair exchanges its columns with
// shuffles, forms alpha = |a_p|^2, beta = |a_q|^2, gamma = a_p . a_q (both
// lanes the same sums in the same order) and, unless |gamma| <= tol
// sqrt(alpha beta), rotates [a_p a_q] (and [v_p v_q]) by the angle that
// makes them orthogonal.  A sweep is 31 rounds; sweeps stop when one rotates
// nothing.  Then A V has orthogonal columns A v_j = lambda_j v_j (A is PSD),
// so lambda_j = |column j| and v_j = column j of V.  No block barrier: the
// warp works alone.  Lanes past R hold zero columns and never rotate.
//
// Outputs (lane j < R writes its own entries): W[rank_j * R + a] =
// sqrt(lambda_j) v_j[a] for a < R, rank_j the ascending rank of lambda_j
// (a NaN ranks last, ties by index), and lam[rank_j] = lambda_j.
//
// A holds the matrix times 2^k (k even, chosen by the caller so that its
// largest entry is near 1: the squared column norms stay inside the FP32
// range); the outputs are scaled back: lambda 2^-k, W rows 2^(-k/2).
__device__ inline void warp_jacobi_psd32(const float *A, int R, int k, double *W, double *lam, int lane) {
    float a[32], v[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        a[i] = (i < R && lane < R) ? A[i * R + lane] : 0.0f;
        v[i] = i == lane ? 1.0f : 0.0f;
    }
    const float tol = FTL_CM_JACOBI_TOL * 5.9604645e-08f;  // units of FP32 rounding
    for (int sweep = 0; sweep < 30; ++sweep) {
        bool rotated = false;
        for (int r = 0; r < 31; ++r) {
            const int partner = lane == 31 ? r : (lane == r ? 31 : (2 * r - lane + 31) % 31);
            float b[32];
            float own = 0.0f, g = 0.0f;
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                b[i] = __shfl_sync(0xffffffffu, a[i], partner);
                own = fmaf(a[i], a[i], own);
            }
            const bool lo = lane < partner;
            // gamma summed in the same order by both lanes: p's entry first
#pragma unroll
            for (int i = 0; i < 32; ++i) g = lo ? fmaf(a[i], b[i], g) : fmaf(b[i], a[i], g);
            const float oth = __shfl_sync(0xffffffffu, own, partner);
            const float ap = lo ? own : oth, aq = lo ? oth : own;
            bool rot = g != 0.0f && fabsf(g) > tol * sqrtf(ap * aq);
            float c = 1.0f, s = 0.0f;
            if (rot) {
                const float zeta = (aq - ap) / (2.0f * g);
                const float t = (zeta >= 0.0f ? 1.0f : -1.0f) / (fabsf(zeta) + sqrtf(1.0f + zeta * zeta));
                c = 1.0f / sqrtf(1.0f + t * t);
                s = c * t;
            }
            rotated |= rot;
            // p: c a_p - s a_q;  q: s a_p + c a_q  (both lanes of a pair
            // rotate or neither: rot is computed from the same values)
            const float cs_own = c, cs_oth = lo ? -s : s;
            if (__any_sync(0xffffffffu, rot)) {
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    const float vb = __shfl_sync(0xffffffffu, v[i], partner);
                    if (rot) {
                        a[i] = fmaf(cs_own, a[i], cs_oth * b[i]);
                        v[i] = fmaf(cs_own, v[i], cs_oth * vb);
                    }
                }
            }
        }
        if (!__any_sync(0xffffffffu, rotated)) break;
    }
    float nrm = 0.0f;
#pragma unroll
    for (int i = 0; i < 32; ++i) nrm = fmaf(a[i], a[i], nrm);
    float lv = sqrtf(nrm);
    if (lv != lv) lv = INFINITY;
    int rank = 0;
    for (int u = 0; u < R; ++u) {
        const float lu = __shfl_sync(0xffffffffu, lv, u);
        if (lu < lv || (lu == lv && u < lane)) ++rank;
    }
    if (lane < R) {
        const double sq = (double)sqrtf(fmaxf(lv, 0.0f)) * ldexp(1.0, -k / 2);
#pragma unroll
        for (int i = 0; i < 32; ++i)
            if (i < R) W[rank * R + i] = sq * (double)v[i];
        lam[rank] = (double)sqrtf(nrm) * ldexp(1.0, -k);
    }
}

// 1/d for a positive normal FP64 d below 2^1023, by the Newton-Raphson
// iteration for the reciprocal: the mantissa m in [1, 2) is inverted in FP32
// (24 correct bits) and refined by two steps x <- x + x (1 - m x) in FP64
// (each step doubles the correct bits: 48, then past 53), and the exponent is
// restored by an exact power of two.  Other inputs take the IEEE division.
// Its dependent path is a few FP64 operations, shorter than the division's
// on GB300's long-latency FP64 pipe.
__device__ __forceinline__ double rcp_newton(double d) {
    const int hi = __double2hiint(d), lo = __double2loint(d);
    const int ef = (hi >> 20) & 0x7ff;
    if (hi < 0 || ef == 0 || ef >= 2046) return 1.0 / d;
    const double m = __hiloint2double((hi & 0x000fffff) | (1023 << 20), lo);
    double x = (double)(1.0f / (float)m);
    double e = fma(-m, x, 1.0);
    x = fma(x, e, x);
    e = fma(-m, x, 1.0);
    x = fma(x, e, x);
    return x * __hiloint2double((2046 - ef) << 20, 0);
}

// Inverse of a symmetric positive definite A (dense R x R FP64 in shared
// memory, upper triangle used, R <= 32) by the sweep operator (Goodnight,
// "A tutorial on the SWEEP operator", The American Statistician 33, 1979):
// sweeping pivot k with d = a_kk and r = 1/d sets
//   a_kk <- -r,  a_kj <- a_kj r,  a_ik <- a_ik r,  a_ij <- a_ij - (a_ik r) a_kj,
// keeps the matrix symmetric, and after all R pivots leaves -A^-1.  The
// pivots of an SPD matrix are its Schur complements, all positive.  Only the
// R(R+1)/2 upper entries are stored and updated, at most two per thread
// (blockDim.x * 2 >= R(R+1)/2), with two FP64 operations per entry and step
// (GB300's FP64 pipe retires two lanes per cycle per SM: every FP64
// instruction a warp issues holds it for 16 cycles).  At each step warp 0
// copies row k (a_kj = a_jk, half of it a strided column of the upper
// triangle) into a contiguous buffer, so the bulk update reads its operands
// without shared-memory bank conflicts, and lane 0 forms the pivot's
// reciprocal (rcp_newton).  On return (true) the upper triangle holds -A^-1;
// false (block-uniformly) when a pivot is not positive.  scratch: R + 1
// doubles; flag: one int.
__device__ inline bool sweep_inverse_spd(double *A, int R, double *scratch, int *flag) {
    const int tid = threadIdx.x, nth = blockDim.x, nup = R * (R + 1) / 2;
    double *row = scratch + 1;
    int oi[2], oj[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        int w = tid + q * nth;
        oi[q] = -1;
        oj[q] = -1;
        if (w < nup) {
            int i = 0;
            while (w >= R - i) {
                w -= R - i;
                ++i;
            }
            oi[q] = i;
            oj[q] = i + w;
        }
    }
    for (int k = 0; k < R; ++k) {
        if (tid < 32) {
            if (tid < R) row[tid] = A[min(k, tid) * R + max(k, tid)];
            if (tid == 0) {
                const double d = A[k * R + k];
                *flag = d > 0.0 ? 1 : 0;
                scratch[0] = d > 0.0 ? rcp_newton(d) : 0.0;
            }
        }
        __syncthreads();
        if (*flag == 0) return false;
        const double r = scratch[0];
        double nv[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            nv[q] = 0.0;
            const int i = oi[q], j = oj[q];
            if (i < 0) continue;
            if (i == k) {
                nv[q] = (j == k) ? -r : row[j] * r;
            } else if (j == k) {
                nv[q] = row[i] * r;
            } else {
                nv[q] = fma(-(row[i] * r), row[j], A[i * R + j]);
            }
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 2; ++q)
            if (oi[q] >= 0) A[oi[q] * R + oj[q]] = nv[q];
        __syncthreads();
    }
    return true;
}

// Block Cholesky pivots through rsqrt (one library call: l = d rsqrt(d), 1/l
// = rsqrt(d)) instead of a square root and a division: a shorter dependent
// FP64 path per step (measured 146k -> 129k cycles for the R = 32 factor and
// inverse in one CTA).
#ifndef FTL_CHOL_RSQRT
#define FTL_CHOL_RSQRT 1
#endif

// In-place lower Cholesky factor of (A - shift I), A dense R x R FP64 in
// shared memory (lower triangle used).  Returns true (block-uniformly) when
// every pivot is positive, i.e. A - shift I is positive definite.  The column
// below a pivot is scaled by the pivot's reciprocal (one FP64 division per
// step instead of one per entry); rinv is one shared-memory double of scratch
// (no static shared memory here: the callers' kernels opt in to the whole
// 227 KB as dynamic shared memory).
__device__ inline bool cholesky_lower(double *A, int R, double shift, int *flag, double *rinv) {
    const int tid = threadIdx.x, nth = blockDim.x;
    if (tid == 0) *flag = 1;
    for (int e = tid; e < R; e += nth) A[e * R + e] -= shift;
    __syncthreads();
    for (int k = 0; k < R; ++k) {
        if (tid == 0) {
            double d = A[k * R + k];
            if (!(d > 0.0)) *flag = 0;
#if FTL_CHOL_RSQRT
            const double r = d > 0.0 ? rsqrt(d) : 1.0;
            A[k * R + k] = d > 0.0 ? d * r : 1.0;
            *rinv = r;
#else
            const double l = d > 0.0 ? sqrt(d) : 1.0;
            A[k * R + k] = l;
            *rinv = 1.0 / l;
#endif
        }
        __syncthreads();
        if (*flag == 0) break;
        const double r = *rinv;
        for (int i = k + 1 + tid; i < R; i += nth) A[i * R + k] *= r;
        __syncthreads();
        const int m = R - k - 1;
        for (int w = tid; w < m * m; w += nth) {
            int i = k + 1 + w / m, jj = k + 1 + w % m;
            if (jj <= i) A[i * R + jj] -= A[i * R + k] * A[jj * R + k];
        }
        __syncthreads();
    }
    __syncthreads();
    return *flag != 0;
}

}  // namespace ftl
