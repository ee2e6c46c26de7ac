// integrator_team.cuh -- the FP32-mixed form with one chain per TEAM of T
// warps (T = 1, 2, 4, 8), for chains of up to 64*T beads. Each team claims
// chains from the device work queue and owns one chain at a time; team thread
// u owns beads u and u + 32T, holding their positions, forces and noise in
// registers. There is no block-wide barrier: neighbour data (bonds, prefix
// sums) goes through the team's own shared-memory area under the team barrier
// (__syncwarp for T = 1, a named barrier otherwise); reductions are warp
// shuffles followed, for T > 1, by a fixed-order sum over the team's warps.
//
// Precision (the mixed form): D.x recomputed pairwise in FP32 from shared FP32
// bead coordinates, FP32 excluded volume and Chebyshev recurrence; FP64
// positions, spring/bending forces, connector solve, Lanczos vectors and
// tridiagonal bounds, and the (rare) Cholesky fallback. The noise stream is
// the reference's ran_1 stream bit for bit, drawn by all team threads at once
// with a jump-ahead (GF(2) powers of the xorshift step, powers of 16807 mod
// 2^31-1).
//
// Reference: src/integrator.cpp:61-170 of the bdsim project and the physics it
// calls; each stage cites its reference function.
#pragma once

#include "integrator.cuh"
#include "team_layout.h"

namespace bdcu {

__device__ __forceinline__ double wsum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    return v;
}

// Barrier over one team: __syncwarp for a single warp, else named barrier
// 1 + team (barrier 0 is __syncthreads') over the team's 32T threads.
template <int T>
__device__ __forceinline__ void team_sync(int team) {
    if constexpr (T == 1) {
        __syncwarp();
    } else {
        asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "r"(32 * T) : "memory");
    }
}

// Number of eigenvalues of the tridiagonal (a, b) below x, from the signs of
// the leading principal minors p_i = (a_i - x) p_{i-1} - b_{i-1}^2 p_{i-2}
// (divide-free Sturm sequence, rescaled against overflow). The mixed form
// uses it in place of sturm_count (src/hydrodynamics.cpp:91-104).
__device__ __forceinline__ int sturm_count_products(const double* a, const double* b, int m, double x) {
    double pm = 1.0, p = a[0] - x;
    int count = (p < 0.0) ? 1 : 0;
    for (int i = 1; i < m; ++i) {
        const double pn = (a[i] - x) * p - b[i - 1] * b[i - 1] * pm;
        count += ((pn < 0.0) != (p < 0.0)) ? 1 : 0;
        pm = p;
        p = pn;
        if (fabs(p) > 1e150) {
            p *= 1e-150;
            pm *= 1e-150;
        }
    }
    return count;
}

// Bisection for the target-th eigenvalue boundary on a half warp (16 lanes,
// depth-4 speculative tree), the iteration of src/hydrodynamics.cpp:196-207.
static __device__ void halfwarp_bisect(const double* al, const double* bb, int k, int target, double& lo, double& hi) {
    const int lane = threadIdx.x & 15;
    const int lvl = 31 - __clz(lane + 1);
    const int p = lane + 1 - (1 << lvl);
    for (int it = 0; it < 100; it += 4) {
        int dec = 0;
        if (lane < 15) {
            double a = lo, b = hi;
            for (int l = 0; l < lvl; ++l) {
                const int bit = (p >> (lvl - 1 - l)) & 1;
                const double m = 0.5 * (a + b);
                if (bit == 0) b = m; else a = m;
            }
            const double mid = 0.5 * (a + b);
            dec = (sturm_count_products(al, bb, k, mid) >= target) ? 0 : 1;
        }
        int node = 0;
        double na = lo, nb = hi;
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            const int d = __shfl_sync(kFull, dec, node, 16);
            const double m = 0.5 * (na + nb);
            if (d == 0) nb = m; else na = m;
            node = 2 * node + 1 + d;
        }
        // settled: the interval stopped shrinking or is within 1e-10 relative
        // (the bounds are padded by 2x / 2% downstream)
        const bool done = (na == lo && nb == hi) || (nb - na) <= 1e-10 * fmax(fabs(na), fabs(nb));
        lo = na;
        hi = nb;
        if (__all_sync(kFull, done)) break;
    }
}

// Eigenvalues below x of a tridiagonal of up to kLanczosWarm entries in
// registers (a; b2: squared off-diagonals): the signs of the leading principal
// minors p_i = (a_i - x) p_{i-1} - b_{i-1}^2 p_{i-2}. |a_i - x| and b^2 lie
// within [1e-20, (3N)^2] or are zero, so eight factors neither overflow nor
// vanish.
__device__ __forceinline__ int sturm_count8(const double (&a)[kLanczosWarm], const double (&b2)[kLanczosWarm], int k,
                                            double x) {
    double pm = 1.0, p = a[0] - x;
    int count = p < 0.0;
#pragma unroll
    for (int i = 1; i < kLanczosWarm; ++i) {
        const double pn = fma(a[i] - x, p, -(b2[i - 1] * pm));
        count += i < k && ((pn < 0.0) != (p < 0.0));
        pm = p;
        p = pn;
    }
    return count;
}

// Multisection for the target-th eigenvalue boundary on a half warp: 15 lanes
// evaluate the Sturm count at 15 evenly spaced interior points of [lo, hi], a
// ballot finds the sixteenth that holds the boundary (4 bits per round), the
// iteration of src/hydrodynamics.cpp:196-207 in place of its halvings. Every
// lane of the half warp ends with the same lo, hi.
__device__ __forceinline__ void halfwarp_multisect(const double (&a)[kLanczosWarm], const double (&b2)[kLanczosWarm],
                                                   int k, int target, double& lo, double& hi) {
    const int h = threadIdx.x & 15;
    const int shift = threadIdx.x & 16;
    for (int it = 0; it < 25; ++it) {
        const double w = hi - lo;
        const bool ge = h < 15 && sturm_count8(a, b2, k, lo + w * ((double)(h + 1) * 0.0625)) >= target;
        const unsigned bal = (__ballot_sync(kFull, ge) >> shift) & 0xffffu;
        const int f = bal ? __ffs(bal) - 1 : 15;
        const double nlo = f == 0 ? lo : lo + w * ((double)f * 0.0625);
        const double nhi = f == 15 ? hi : lo + w * ((double)(f + 1) * 0.0625);
        // settled: the interval stopped shrinking or is within 1e-6 relative
        // (the bounds are padded by 2x / 2% downstream, and the FD check
        // polices the Chebyshev result)
        const bool done = (nlo == lo && nhi == hi) || (nhi - nlo) <= 1e-6 * fmax(fabs(nlo), fabs(nhi));
        lo = nlo;
        hi = nhi;
        if (__all_sync(kFull, done)) break;
    }
}

// m x mod 2^31 - 1, by folding the product's high part onto the low one.
__device__ __forceinline__ uint32_t lehmer_mul(uint32_t m, uint32_t x) {
    const uint64_t p = (uint64_t)m * x;
    const uint32_t r = (uint32_t)(p & 0x7fffffffu) + (uint32_t)(p >> 31);
    return r >= 0x7fffffffu ? r - 0x7fffffffu : r;
}
// The xorshift state x advanced by the matrix power whose columns are given.
__device__ __forceinline__ uint32_t xorshift_jump(const uint32_t* cols, uint32_t x) {
    uint32_t y = 0;
#pragma unroll 8
    for (int i = 0; i < 32; ++i) y ^= cols[i] & (0u - ((x >> i) & 1u));
    return y;
}

// 1/x for |x| in [1e-30, 1e30]: a single-precision seed refined by two
// Newton-Raphson steps r <- r (2 - x r) (quadratic convergence: 2^-23 ->
// 2^-46 -> below double rounding).
__device__ __forceinline__ double rcp_newton(double x) {
    float f;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(f) : "f"((float)x));
    double r = (double)f;
    r = r * (2.0 - x * r);
    r = r * (2.0 - x * r);
    return r;
}

// Inverse iteration for a Ritz vector (src/hydrodynamics.cpp:106-136) with the
// tridiagonal (k <= kLanczosWarm) in registers; every lane that calls it
// computes the same y. kPasses: the reference's two in the plain form (a
// single solve closer to the eigenvalue leaves 1e-10 of the other vectors, two
// at 1e-7 leave 1e-15); one in the mixed form, whose shift is within 1e-6
// relative of the eigenvalue, so a single solve already amplifies its
// eigenvector by ~1e5 over the others (the vector only seeds the next step's
// Lanczos).
template <int kPasses>
__device__ __forceinline__ void tridiag_vec_reg(const double (&a)[kLanczosWarm], const double (&b)[kLanczosWarm],
                                                int m, double lambda, double (&y)[kLanczosWarm]) {
    const double scale = dmax_(fabs(lambda), 1.0);
    const double shift = lambda - 1.0e-7 * scale;
    const double y0 = rsqrt((double)m);
    double c[kLanczosWarm];
#pragma unroll
    for (int i = 0; i < kLanczosWarm; ++i) y[i] = i < m ? y0 : 0.0;
#pragma unroll 1
    for (int it = 0; it < kPasses; ++it) {
        // pivots: the reference's tiny-pivot guard (1e-300) raised to 1e-30 so
        // that the reciprocal's single-precision seed stays in range (the
        // vector only seeds the next step's Lanczos)
        double beta = a[0] - shift;
        if (fabs(beta) < 1.0e-30) beta = 1.0e-30;
        double ib = rcp_newton(beta);
        c[0] = (m > 1 ? b[0] * ib : 0.0);
        y[0] = y[0] * ib;
#pragma unroll
        for (int i = 1; i < kLanczosWarm; ++i) {
            if (i < m) {
                beta = (a[i] - shift) - b[i - 1] * c[i - 1];
                if (fabs(beta) < 1.0e-30) beta = 1.0e-30;
                ib = rcp_newton(beta);
                c[i] = (i < m - 1 ? b[i] * ib : 0.0);
                y[i] = (y[i] - b[i - 1] * y[i - 1]) * ib;
            }
        }
#pragma unroll
        for (int i = kLanczosWarm - 2; i >= 0; --i)
            if (i < m - 1) y[i] = y[i] - c[i] * y[i + 1];
        double nrm = 0.0;
#pragma unroll
        for (int i = 0; i < kLanczosWarm; ++i) nrm += y[i] * y[i];
        nrm = sqrt(nrm);
        if (!(nrm > 0.0) || !isfinite(nrm)) {
#pragma unroll
            for (int i = 0; i < kLanczosWarm; ++i) y[i] = i < m ? y0 : 0.0;
            return;
        }
        const double inr = 1.0 / nrm;
#pragma unroll
        for (int i = 0; i < kLanczosWarm; ++i) y[i] *= inr;
    }
}

// Inverse iteration for a Ritz vector (src/hydrodynamics.cpp:106-136), one lane.
static __device__ void wk_tridiag_vec(const double* a, const double* b, int m, double lambda, double* y, double* c,
                                      double* d) {
    const double scale = dmax_(fabs(lambda), 1.0);
    const double shift = lambda - 1.0e-7 * scale;
    const double y0 = rsqrt((double)m);
    for (int i = 0; i < m; ++i) y[i] = y0;
    for (int it = 0; it < 2; ++it) {
        double beta0 = a[0] - shift;
        if (fabs(beta0) < 1.0e-300) beta0 = 1.0e-300;
        double ib = 1.0 / beta0;
        c[0] = (m > 1 ? b[0] * ib : 0.0);
        d[0] = y[0] * ib;
        for (int i = 1; i < m; ++i) {
            double beta = (a[i] - shift) - b[i - 1] * c[i - 1];
            if (fabs(beta) < 1.0e-300) beta = 1.0e-300;
            ib = 1.0 / beta;
            c[i] = (i < m - 1 ? b[i] * ib : 0.0);
            d[i] = (y[i] - b[i - 1] * d[i - 1]) * ib;
        }
        y[m - 1] = d[m - 1];
        for (int i = m - 2; i >= 0; --i) y[i] = d[i] - c[i] * y[i + 1];
        double nrm = 0.0;
        for (int i = 0; i < m; ++i) nrm += y[i] * y[i];
        nrm = sqrt(nrm);
        if (!(nrm > 0.0) || !isfinite(nrm)) {
            for (int i = 0; i < m; ++i) y[i] = y0;
            return;
        }
        const double inr = 1.0 / nrm;
        for (int i = 0; i < m; ++i) y[i] *= inr;
    }
}

// Which vectors of a cold Lanczos run are projected on the whole basis (the reference
// projects every one, src/hydrodynamics.cpp:146-264): a bound on their loss of
// orthogonality, carried along by the recurrence that the loss follows (H. D. Simon,
// "The Lanczos algorithm with partial reorthogonalization", Math. Comp. 42, 1984),
//   |v_{j+1}.v_i| <= ((|a_i - a_j| + b_i + b_{i+1}) w_j + b_j w_{j-1} + eps |D|) / b_{j+1}
// with the largest factor over i. Once it passes `tol` two consecutive vectors are
// projected, as both enter the recurrence. tol is the square root of the products'
// rounding, up to which the tridiagonal is the projection of D to that rounding, with
// a margin. b_{j+1} comes from |D v_j|^2 by Pythagoras; where that cancels (below
// `tiny` of it) the vectors are projected in any case. (Two of every six, whatever the
// spectrum, lost all orthogonality within four steps on chains whose beads lie close
// together: bounds off by up to 18x in FP64 and 1e4x on FP32 products. Projected:
// 20% of the vectors on coils and 32% on collapsed chains, 39 and 56% on FP32 products.)
// FP32 but for the cancelling difference: the bound's latency is on every step's path.
struct BasisLoss {
    float w = 0.f, wp = 0.f, lo = 0.f, hi = 0.f, bmax = 0.f;
    bool again = false;
    // After step j's alpha, beta (none at j = 0) and ww = |D v_j|^2: project the next vector?
    __device__ __forceinline__ bool project(int j, double al, double bt, double ww, float eps, float tol, float tiny) {
        if (j == 0) {
            lo = hi = (float)al;
            bt = 0.0;
        }
        const float a = (float)al, b = (float)bt, sq = (float)fma(-bt, bt, fma(-al, al, ww));
        lo = fminf(lo, a);
        hi = fmaxf(hi, a);
        bmax = fmaxf(bmax, b);
        const bool lost = !(sq > tiny * (float)ww);
        const float ib = lost ? 1.f : rsqrtf(sq), bn = lost ? 1.f : sq * ib;
        const float f = fmaxf(hi - a, a - lo) + 2.f * fmaxf(bmax, bn);
        float wn = (f * w + b * wp + eps * (fabsf(a) + b + bn)) * ib;
        const bool hit = lost || !(wn <= tol), now = hit || again;
        again = lost || (hit && !again);
        if (now) wn = eps;
        wp = w;
        w = wn;
        return now;
    }
};

// Right-looking Cholesky factor (cholesky_lower, src/linalg.cpp:91-107) of the n x n
// matrix at L in global scratch, by a team of T warps. Returns false if not positive
// definite. The trailing update takes eight columns at a time, so that a thread's
// loads of one row segment are in flight together: the cached pair weights leave
// little of an SM's memory as L1, and a column by itself waits for L2 (N = 50:
// 1.3 ms a factor while it stayed in L1, 2.9 from L2, 0.92 so).
template <int T>
static __device__ __noinline__ bool team_factor(double* L, int n, int tid, int team) {
    constexpr int TT = 32 * T, kCols = 8;
    for (int k = 0; k < n; ++k) {
        double* colk = L + (int64_t)k * n;
        const double s = colk[k];
        if (!(s > 0.0)) return false;
        const double dk = sqrt(s);
        team_sync<T>(team);
        if (tid == 0) colk[k] = dk;
        const double idk = 1.0 / dk;
        for (int i = k + 1 + tid; i < n; i += TT) colk[i] *= idk;
        __threadfence_block();
        team_sync<T>(team);
        for (int j = k + 1; j < n; j += kCols) {
            double l[kCols];
#pragma unroll
            for (int u = 0; u < kCols; ++u) l[u] = colk[min(j + u, n - 1)];
            for (int i = j + tid; i < n; i += TT) {
                const double c = colk[i];
                double v[kCols];
#pragma unroll
                for (int u = 0; u < kCols; ++u) v[u] = i >= j + u ? L[(int64_t)(j + u) * n + i] : 0.0;
#pragma unroll
                for (int u = 0; u < kCols; ++u)
                    if (i >= j + u) L[(int64_t)(j + u) * n + i] = fma(-c, l[u], v[u]);
            }
        }
        __threadfence_block();
        team_sync<T>(team);
    }
    return true;
}

template <int T, int Q>
struct TeamChain {
    static constexpr int TT = 32 * T;  // threads of the team
    const RunArgs& a;
    TeamShared<T, Q>& S;
    const DevChain& ch;
    double* V;      // warm Lanczos basis in shared memory (kLanczosWarm x nv)
    float* sqx;     // Chebyshev node values, aliasing V (dead after the bounds)
    float* coef;    // Chebyshev coefficients, aliasing V
    float* ct;      // cosine table, aliasing V
    double* Vg;     // cold basis in global scratch (kLanczosCold x nv)
    double* Lt;     // Cholesky factor in global scratch (n x n)
    int nv;
    int tid;        // thread in the team
    int wl, wi;     // lane in its warp, warp in the team
    int team;       // team in the thread block (named barrier 1 + team)
    int N, n;
    bool hi;
    float4* Wt;     // cached pair weights (omega1 of j, j+1, omega2 of j, j+1): row j/2, column bead
    int jc;         // partner beads below jc have cached weights (a multiple of four)
    int par, xpar;  // parity of the reduction buffer and of the single products' input rows
    int32_t cnt[8];  // this call's counts for the chain (added to the 64-bit counters at the end)
    int status;
    // RPY constants (FP32). Bead coordinates are staged divided by `scale`
    // (= h* under HI), which turns the RPY weights into functions of
    // rho = h*/r alone.
    float scale, iscale, K1, K2, K3, C3, C7;

    __device__ TeamChain(const RunArgs& a_, TeamShared<T, Q>& S_, const DevChain& ch_) : a(a_), S(S_), ch(ch_) {}

    __device__ __forceinline__ bool valid(int q) const { return tid + TT * q < N; }
    __device__ __forceinline__ int bead(int q) const { return tid + TT * q; }
    __device__ __forceinline__ void sync() const { team_sync<T>(team); }

    // Sums over the team, the same bits in every thread: warp butterflies, then
    // the warps' partial sums added in warp order. One barrier: consecutive
    // calls alternate between two buffers.
    __device__ __forceinline__ double* next_red() {
        double* r = S.red[par];
        par ^= 1;
        return r;
    }
    template <int M>
    __device__ __forceinline__ void sums(double (&v)[M]) {
#pragma unroll
        for (int m = 0; m < M; ++m) v[m] = wsum(v[m]);
        if constexpr (T > 1) {
            double* r = next_red();
            if (wl == 0)
#pragma unroll
                for (int m = 0; m < M; ++m) r[m * T + wi] = v[m];
            sync();
#pragma unroll
            for (int m = 0; m < M; ++m) {
                v[m] = r[m * T];
#pragma unroll
                for (int w = 1; w < T; ++w) v[m] += r[m * T + w];
            }
        }
    }
    __device__ __forceinline__ double tsum(double v) {
        double a1[1] = {v};
        sums(a1);
        return a1[0];
    }

    // Eight sums over the warp at once: halves of the vector exchanged with
    // lanes ^16, ^8, ^4, then a butterfly over ^2, ^1; value u ends in lanes
    // 4u..4u+3, which publish it for their warp at out[u * T + warp].
    __device__ __forceinline__ void warp_sum8(const double (&c)[8], double* out) const {
        const bool u16 = wl & 16, u8 = wl & 8, u4 = wl & 4;
        double k4[4], k2[2];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            k4[u] = (u16 ? c[u + 4] : c[u]) + __shfl_xor_sync(kFull, u16 ? c[u] : c[u + 4], 16);
#pragma unroll
        for (int u = 0; u < 2; ++u)
            k2[u] = (u8 ? k4[u + 2] : k4[u]) + __shfl_xor_sync(kFull, u8 ? k4[u] : k4[u + 2], 8);
        double t = (u4 ? k2[1] : k2[0]) + __shfl_xor_sync(kFull, u4 ? k2[0] : k2[1], 4);
        t += __shfl_xor_sync(kFull, t, 2);
        t += __shfl_xor_sync(kFull, t, 1);
        if ((wl & 3) == 0) out[(wl >> 2) * T + wi] = t;
    }
    // After a barrier: the total over the warps of published value u.
    __device__ __forceinline__ double total(const double* r, int u) const {
        double t = r[u * T];
#pragma unroll
        for (int w = 1; w < T; ++w) t += r[u * T + w];
        return t;
    }

    // OR of status bits over the team.
    __device__ int tor(int v) {
        v = __reduce_or_sync(kFull, v);
        if constexpr (T == 1) {
            return v;
        } else {
            sync();
            if (wl == 0) S.flag[wi] = v;
            sync();
            int s = 0;
#pragma unroll
            for (int w = 0; w < T; ++w) s |= S.flag[w];
            return s;
        }
    }

    // ---- FP32 matrix-free D.x (Diffusion::apply, src/mobility.cpp:53-56;
    // RPY weights src/hydrodynamics.cpp:36-43). x, y: the thread's beads.
    // K products against the same D in one pass over the bead pairs: the
    // pair geometry and weights are computed once for all K inputs (K = 3
    // for the products of a step that do not depend on one another).
    //
    // The partner beads j are taken two at a time in packed FP32x2 arithmetic
    // (sm_100's FADD2 / FMUL2 / FFMA2: one issue slot for the pair; the FP32 pipe
    // rate is that of scalar FFMA, measured 73 TFLOP/s on one B200 either way),
    // from coordinates and inputs staged by component in shared memory, so
    // one 64-bit broadcast load brings (j, j+1) of a component. Each bead's
    // sum is kept as two interleaved partial sums (even and odd j), added at
    // the end. N is padded to a multiple of four with zero inputs (whose
    // contribution om1 * 0 + om2 (d . 0) d is exactly zero).
    // The pair weights of the first jc partner beads are computed once a step
    // (build_weights) and kept in shared memory, 8 bytes per pair: a product
    // then takes 13 packed operations per bead and two partners instead of about
    // 35, and a chain of dependent operations half as long. The rest, where
    // they do not fit (N above about 100), are evaluated in every product by the
    // same operations, so a result does not depend on jc.
    template <int K>
    __device__ __forceinline__ void applyK(const float (&x)[K][Q][3], float (&acc)[K][Q][3]) {
        static_assert(K >= 1 && K <= 3, "applyK stages at most three inputs");
        cnt[C_DX] += K;
        // single products alternate between input rows 0 and 1, so that the
        // barrier after staging also guards the rows' next use; the fused sets
        // wait for the products before them
        float(*xr)[3][32 * T * Q] = S.xk;
        if (K == 1) {
            xr += xpar;
            xpar ^= 1;
        } else {
            sync();
        }
#pragma unroll
        for (int q = 0; q < Q; ++q)
            if (valid(q))
#pragma unroll
                for (int r = 0; r < K; ++r)
#pragma unroll
                    for (int d = 0; d < 3; ++d) xr[r][d][bead(q)] = x[r][q][d];
        const int pad = -N & 3;  // zero inputs up to a multiple of four beads
        if (tid < 3 * K * pad) xr[tid / (3 * pad)][tid / pad % 3][N + tid % pad] = 0.f;
        sync();
        bool one_slot = false;
        if constexpr (Q == 2) one_slot = __all_sync(kFull, !valid(1));
        const int nq = one_slot ? 1 : Q;
        float2 nb[Q][3], a[K][Q][3];
        own_coordinates(nb);
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
            for (int d = 0; d < 3; ++d)
#pragma unroll
                for (int r = 0; r < K; ++r) a[r][q][d] = make_float2(0.f, 0.f);
        auto products = [&](int q, const float2& dx, const float2& dy, const float2& dz, const float2& om1,
                            const float2& om2, const float2 (&xj)[K][3]) {
#pragma unroll
            for (int r = 0; r < K; ++r) {
                const float2 tt =
                    __fmul2_rn(om2, __ffma2_rn(dz, xj[r][2], __ffma2_rn(dy, xj[r][1], __fmul2_rn(dx, xj[r][0]))));
                a[r][q][0] = __ffma2_rn(tt, dx, __ffma2_rn(om1, xj[r][0], a[r][q][0]));
                a[r][q][1] = __ffma2_rn(tt, dy, __ffma2_rn(om1, xj[r][1], a[r][q][1]));
                a[r][q][2] = __ffma2_rn(tt, dz, __ffma2_rn(om1, xj[r][2], a[r][q][2]));
            }
        };
        const int n2 = (N + 1) & ~1;
        int j = 0;
        const float4* w = Wt;
        // cached weights: four partner beads per step (the second pair of the
        // last step may lie beyond N: its inputs are zero)
#pragma unroll 1
        for (; j < jc; j += 4, w += 2 * N) {
            float4 pj[3], xj[K][3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                pj[d] = *reinterpret_cast<const float4*>(&S.ps[d][j]);
#pragma unroll
                for (int r = 0; r < K; ++r) xj[r][d] = *reinterpret_cast<const float4*>(&xr[r][d][j]);
            }
#pragma unroll
            for (int q = 0; q < Q; ++q)
                if (q < nq) {
                    const int m = min(bead(q), N - 1);
                    const float4 o[2] = {w[m], w[N + m]};
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        float2 p[3], x2[K][3];
#pragma unroll
                        for (int d = 0; d < 3; ++d) {
                            p[d] = h ? make_float2(pj[d].z, pj[d].w) : make_float2(pj[d].x, pj[d].y);
#pragma unroll
                            for (int r = 0; r < K; ++r)
                                x2[r][d] = h ? make_float2(xj[r][d].z, xj[r][d].w) : make_float2(xj[r][d].x, xj[r][d].y);
                        }
                        products(q, __fadd2_rn(p[0], nb[q][0]), __fadd2_rn(p[1], nb[q][1]), __fadd2_rn(p[2], nb[q][2]),
                                 make_float2(o[h].x, o[h].y), make_float2(o[h].z, o[h].w), x2);
                    }
                }
        }
        // the rest: weights evaluated here
#pragma unroll 1
        for (; j < n2; j += 2) {
            float2 pj[3], xj[K][3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                pj[d] = *reinterpret_cast<const float2*>(&S.ps[d][j]);
#pragma unroll
                for (int r = 0; r < K; ++r) xj[r][d] = *reinterpret_cast<const float2*>(&xr[r][d][j]);
            }
            if (K == 1 && Q == 2 && nq == 2) {
                // both beads' chains of operations side by side, with one branch
                // for their near pairs (N = 500: two warps per scheduler leave
                // the FP32 pipe 46% busy with the beads one after the other)
                float2 d[Q][3], sq[Q], om1[Q], om2[Q];
#pragma unroll
                for (int q = 0; q < Q; ++q) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) d[q][c] = __fadd2_rn(pj[c], nb[q][c]);
                    far_weights2(d[q], sq[q], om1[q], om2[q]);
                }
                if (fminf(fminf(sq[0].x, sq[0].y), fminf(sq[Q - 1].x, sq[Q - 1].y)) < kNear)
#pragma unroll
                    for (int q = 0; q < Q; ++q) near_weights2(sq[q], om1[q], om2[q]);
#pragma unroll
                for (int q = 0; q < Q; ++q) products(q, d[q][0], d[q][1], d[q][2], om1[q], om2[q], xj);
            } else {
#pragma unroll
                for (int q = 0; q < Q; ++q)
                    if (q < nq) {
                        const float2 d[3] = {__fadd2_rn(pj[0], nb[q][0]), __fadd2_rn(pj[1], nb[q][1]),
                                             __fadd2_rn(pj[2], nb[q][2])};
                        float2 om1, om2;
                        pair_weights2(d, om1, om2);
                        products(q, d[0], d[1], d[2], om1, om2, xj);
                    }
            }
        }
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
            for (int d = 0; d < 3; ++d)
#pragma unroll
                for (int r = 0; r < K; ++r) acc[r][q][d] = valid(q) ? a[r][q][d].x + a[r][q][d].y : 0.f;
    }

    // Minus the coordinates of the thread's beads, both halves.
    __device__ __forceinline__ void own_coordinates(float2 (&nb)[Q][3]) const {
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const float v = valid(q) ? -S.ps[d][bead(q)] : 0.f;
                nb[q][d] = make_float2(v, v);
            }
    }

    __device__ __forceinline__ static float rsqrt_approx(float x) {
        float y;
        asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
        return y;
    }

    // RPY weights of two pairs. In units of h*: with d = (R_j - R_b)/h*, s =
    // |d|^2, rho = s^-1/2,
    //   far  (s >= 4 pi): om1 = rho (K1 + K2 rho^2), om2 = rho^3 (K1 - K3 rho^2)
    //   near (s <  4 pi): om1 = 1 - C3 s rho,         om2 = C7 rho
    // and y_b += om1 x_j + om2 (d.x_j) d. The far weights are computed for all,
    // the near ones in a branch that only neighbours along the chain and close
    // contacts take. The self pair (d = 0, s clamped to 1e-24) is a near one
    // with om1 = 1 exactly in FP32 and om2 d = 0: the identity block.
    static constexpr float kNear = 12.566370614359172f;  // 4 pi
    __device__ __forceinline__ void far_weights2(const float2 (&d)[3], float2& sq, float2& om1, float2& om2) const {
        const float2 k1 = make_float2(K1, K1), k2 = make_float2(K2, K2), mk3 = make_float2(-K3, -K3);
        sq = __ffma2_rn(d[2], d[2], __ffma2_rn(d[1], d[1], __fmul2_rn(d[0], d[0])));
        const float2 rho = make_float2(rsqrt_approx(sq.x), rsqrt_approx(sq.y));
        const float2 t = __fmul2_rn(rho, rho);
        om1 = __fmul2_rn(rho, __ffma2_rn(k2, t, k1));
        om2 = __fmul2_rn(__fmul2_rn(rho, t), __ffma2_rn(mk3, t, k1));
    }
    __device__ __forceinline__ void near_weights2(const float2& sq, float2& om1, float2& om2) const {
        const float2 sc = make_float2(fmaxf(sq.x, 1e-24f), fmaxf(sq.y, 1e-24f));
        const float2 rc = make_float2(rsqrt_approx(sc.x), rsqrt_approx(sc.y));
        const float2 n1 = __ffma2_rn(make_float2(-C3, -C3), __fmul2_rn(sc, rc), make_float2(1.f, 1.f));
        const float2 n2 = __fmul2_rn(make_float2(C7, C7), rc);
        om1 = make_float2(sq.x < kNear ? n1.x : om1.x, sq.y < kNear ? n1.y : om1.y);
        om2 = make_float2(sq.x < kNear ? n2.x : om2.x, sq.y < kNear ? n2.y : om2.y);
    }
    __device__ __forceinline__ void pair_weights2(const float2 (&d)[3], float2& om1, float2& om2) const {
        float2 sq;
        far_weights2(d, sq, om1, om2);
        if (fminf(sq.x, sq.y) < kNear) near_weights2(sq, om1, om2);
    }

    // Weights of the thread's beads with partners below jc at the staged
    // positions. Each thread reads back only its own columns (no barrier).
    __device__ __forceinline__ void build_weights() {
        float2 nb[Q][3];
        own_coordinates(nb);
#pragma unroll 2
        for (int j = 0; j < jc; j += 2) {
            float2 pj[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) pj[d] = *reinterpret_cast<const float2*>(&S.ps[d][j]);
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const float2 d[3] = {__fadd2_rn(pj[0], nb[q][0]), __fadd2_rn(pj[1], nb[q][1]),
                                     __fadd2_rn(pj[2], nb[q][2])};
                float2 om1, om2;
                pair_weights2(d, om1, om2);
                if (valid(q)) Wt[(j >> 1) * N + bead(q)] = make_float4(om1.x, om1.y, om2.x, om2.y);
            }
        }
    }

    __device__ void apply32(const float (&x)[Q][3], float (&acc)[Q][3]) {
        applyK<1>(reinterpret_cast<const float(&)[1][Q][3]>(x), reinterpret_cast<float(&)[1][Q][3]>(acc));
    }

    __device__ void apply(const double (&x)[Q][3], double (&y)[Q][3]) {
        if (!hi) {
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int d = 0; d < 3; ++d) y[q][d] = x[q][d];
            return;
        }
        float xf[Q][3], yf[Q][3];
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
            for (int d = 0; d < 3; ++d) xf[q][d] = (float)x[q][d];
        apply32(xf, yf);
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
            for (int d = 0; d < 3; ++d) y[q][d] = (double)yf[q][d];
    }

    // D.x on FP32 thread vectors (identity without HI).
    __device__ void applyF(const float (&x)[Q][3], float (&y)[Q][3]) {
        if (!hi) {
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int d = 0; d < 3; ++d) y[q][d] = x[q][d];
            return;
        }
        apply32(x, y);
    }

    __device__ double dotf(const float (&x)[Q][3], const float (&y)[Q][3]) {
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
            for (int d = 0; d < 3; ++d) s += (double)x[q][d] * (double)y[q][d];
        return tsum(s);
    }

    __device__ double dot(const double (&x)[Q][3], const double (&y)[Q][3]) {
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
            for (int d = 0; d < 3; ++d) s += x[q][d] * y[q][d];
        return tsum(s);
    }

    __device__ void stage_pos(const double (&R)[Q][3]) {
        sync();
#pragma unroll
        for (int q = 0; q < Q; ++q)
            if (valid(q)) {
                const float x = (float)(R[q][0] * iscale), y = (float)(R[q][1] * iscale), z = (float)(R[q][2] * iscale);
                S.pos[bead(q)] = make_float4(x, y, z, 0.f);
                S.ps[0][bead(q)] = x;
                S.ps[1][bead(q)] = y;
                S.ps[2][bead(q)] = z;
            }
        const int pad = -N & 3;  // pad beads (zero input in every pass)
        if (tid < 3 * pad) S.ps[tid / pad][N + tid % pad] = 0.f;
        sync();
    }

    __device__ void to_smem(double* buf, const double (&x)[Q][3]) const {
#pragma unroll
        for (int q = 0; q < Q; ++q)
            if (valid(q))
#pragma unroll
                for (int d = 0; d < 3; ++d) buf[3 * bead(q) + d] = x[q][d];
    }

    // ---- forces at R (FP64 springs/bending/external, FP32 EV) ------------
    // Fs: spring bead forces (src/spring.cpp:195-207). Fe: (EV + bending) +
    // external(t) (src/model.hpp:56-64). Positions must be staged (S.pos).
    __device__ void forces(const double (&R)[Q][3], double t, float (&Fs)[Q][3], float (&Fe)[Q][3], bool spring) {
        const bool bend = ch.bend_type != BDCU_BEND_NONE && N > 2;
        const bool bonds = spring || bend;  // bond forces, unit bonds, lengths: springs and bending only
        if (bonds) to_smem(S.s0, R);
        sync();
        // bonds b = bead(0), bead(1) (b < N-1): Fc -> s1, unit bonds -> s2, lengths -> s3
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const int b = bead(q);
            if (bonds && b < N - 1) {
                const double b0 = S.s0[3 * b + 3] - S.s0[3 * b], b1 = S.s0[3 * b + 4] - S.s0[3 * b + 1],
                             b2 = S.s0[3 * b + 5] - S.s0[3 * b + 2];
                const double len = clamped_len(b0, b1, b2);
                const double f = connector_factor(ch, len);
                S.s1[3 * b] = f * b0;
                S.s1[3 * b + 1] = f * b1;
                S.s1[3 * b + 2] = f * b2;
                const double il = 1.0 / len;
                S.s2[3 * b] = il * b0;
                S.s2[3 * b + 1] = il * b1;
                S.s2[3 * b + 2] = il * b2;
                S.s3[b] = len;
            }
        }
        sync();
        if (bend) {
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const int b = bead(q);
                if (b < N - 2)
                    S.s4[b] = S.s2[3 * (b + 1)] * S.s2[3 * b] + S.s2[3 * (b + 1) + 1] * S.s2[3 * b + 1] +
                              S.s2[3 * (b + 1) + 2] * S.s2[3 * b + 2];
            }
            sync();
        }
        // EV on the scaled coordinates: r = scale*|d|, force -fac(r) * scale * d
        const float zs = (float)(ch.zsbyds5 * scale), p5 = (float)(ch.pt5bydssq * (double)scale * scale);
        // excluded volume, FP32 pair sums over both bead slots at once: the
        // force on m from j is -fac(r) (R_j - R_m), |j - m| >= contour distance
        float fev[Q][3] = {};
        if (ch.ev_type == BDCU_EV_GAUSS) {
            float4 pm[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q) pm[q] = valid(q) ? S.pos[bead(q)] : make_float4(0.f, 0.f, 0.f, 0.f);
            const int cd = ch.cd;
#pragma unroll 4
            for (int j = 0; j < N; ++j) {
                const float4 pj = S.pos[j];
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    const int m = bead(q);
                    const float dx = pj.x - pm[q].x, dy = pj.y - pm[q].y, dz = pj.z - pm[q].z;
                    const float sq = dx * dx + dy * dy + dz * dz;
                    const int dj = j > m ? j - m : m - j;
                    const float fac = ((dj >= cd && j != m) ? zs : 0.f) * __expf(-sq * p5);  // (no branch)
                    fev[q][0] -= fac * dx;
                    fev[q][1] -= fac * dy;
                    fev[q][2] -= fac * dz;
                }
            }
        } else if (ch.ev_type != BDCU_EV_NONE) {
            // LJ and SDK vanish beyond their outer cutoff: pairs outside it are
            // passed over on the FP32 squared distance (a margin of 1e-5 covers
            // its rounding; the cutoff itself is tested in FP64 on r). Each lane
            // meets few partners inside, and the FP64 factor costs a hundred
            // times the test.
            const double* phi = (ch.ev_type == BDCU_EV_SDK && ch.phi_off >= 0) ? a.arena + ch.phi_off : nullptr;
            const double cut = ev_outer_cutoff(ch) * (double)iscale, s2 = (double)scale * scale;
            const float cut2 = (float)(cut * cut * 1.00001);
            float4 pm[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q) pm[q] = valid(q) ? S.pos[bead(q)] : make_float4(3e18f, 3e18f, 3e18f, 0.f);
#pragma unroll 2
            for (int j = 0; j < N; ++j) {
                const float4 pj = S.pos[j];
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    const int m = bead(q);
                    const float dx = pj.x - pm[q].x, dy = pj.y - pm[q].y, dz = pj.z - pm[q].z;
                    const float sq = fmaxf(dx * dx + dy * dy + dz * dz, 1e-12f);
                    const int dj = j > m ? j - m : m - j;
                    if (!(sq <= cut2) || dj < ch.cd || j == m || m >= N) continue;
                    const int mu = j < m ? j : m, nu = j < m ? m : j;
                    const float fac = (float)(ev_factor_short(ch, (double)sq * s2, phi ? phi + (int64_t)mu * N + nu : nullptr) * scale);
                    fev[q][0] -= fac * dx;
                    fev[q][1] -= fac * dy;
                    fev[q][2] -= fac * dz;
                }
            }
        }
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const int m = bead(q);
            if (!valid(q)) {
                for (int d = 0; d < 3; ++d) Fs[q][d] = Fe[q][d] = 0.f;
                continue;
            }
            if (spring) {
                for (int d = 0; d < 3; ++d) {
                    double v;
                    if (m == 0) v = S.s1[d];
                    else if (m == N - 1) v = -S.s1[3 * (N - 2) + d];
                    else v = S.s1[3 * m + d] - S.s1[3 * (m - 1) + d];
                    Fs[q][d] = (float)v;
                }
            }
            double fb[3] = {0.0, 0.0, 0.0}, fx[3] = {0.0, 0.0, 0.0};
            if (bend) bending_on_bead(ch, m, S.s2, S.s4, S.s3, fb);
            if (ch.ext_n > 0) external_on_bead(ch, a.arena, m, t, fx);
            Fe[q][0] = (float)(((double)fev[q][0] + fb[0]) + fx[0]);
            Fe[q][1] = (float)(((double)fev[q][1] + fb[1]) + fx[1]);
            Fe[q][2] = (float)(((double)fev[q][2] + fb[2]) + fx[2]);
        }
        sync();
    }

    // ---- noise: the 3N draws of raw_noise (src/mobility.cpp:18-29) -------
    // The team's threads draw contiguous blocks of c draws of the stream. Each
    // keeps the generator's state at the start of its block: jumped there once
    // per chain with the tabulated powers, and from step to step by the same 3N
    // draws for every thread, so the uniforms equal ran_1's, bit for bit.
    __device__ __forceinline__ void noise_start(uint32_t& ux, int32_t& iy, int32_t& sd) {
        if (sd <= 0 || iy < 0) {
            const int32_t s = sd < 0 ? -sd : sd;
            iy = (888889999 ^ s) | 1;
            ux = (uint32_t)(777755555 ^ s);
            sd = s + 1;
        }
        const int k0 = min(tid * ((n + TT - 1) / TT), n);
        ux = xorshift_jump(a.xs_pow + 32 * (int64_t)k0, ux);
        iy = (int32_t)lehmer_mul(a.a_pow[k0], (uint32_t)iy);
        if (tid < 32) S.jcols[tid] = a.xs_pow[32 * (int64_t)n + tid];
        sync();
    }
    __device__ void noise(uint32_t& ux0, int32_t& iy0, float (&X)[Q][3]) {
        const int c = (n + TT - 1) / TT, k0 = tid * c, k1 = min(n, k0 + c);
        const float am = __fdiv_rn(__int_as_float(0x3f7fffff), 2147483648.0f);
        uint32_t ux = ux0, iy = (uint32_t)iy0;
        for (int k = k0; k < k1; ++k) {
            ux ^= (ux << 13);
            ux ^= (ux >> 17);
            ux ^= (ux << 5);
            iy = lehmer_mul(16807u, iy);
            const int32_t res = (int32_t)(((ux ^ iy) & 0x7fffffffu) | 1u);
            S.s0[k] = (double)__fmul_rn(am, __int2float_rn(res));
        }
        ux0 = xorshift_jump(S.jcols, ux0);
        iy0 = (int32_t)lehmer_mul(a.a_pow[n], (uint32_t)iy0);
        sync();
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                double v = 0.0;
                if (valid(q)) {
                    const double y = S.s0[3 * bead(q) + d] - 0.5;
                    v = (14.14855378 * y * y + 1.21569221) * y;
                }
                X[q][d] = (float)v;
            }
        sync();
    }

    // ---- Lanczos extreme eigenvalues (src/hydrodynamics.cpp:146-264) ----
    __device__ double* basis(int j, int m) { return (m <= kLanczosWarm ? V : Vg) + (int64_t)j * nv; }
    __device__ void load(const double* vec, double (&x)[Q][3]) const {
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
            for (int d = 0; d < 3; ++d) x[q][d] = valid(q) ? vec[3 * bead(q) + d] : 0.0;
    }
    __device__ void store(double* vec, const double (&x)[Q][3]) const {
#pragma unroll
        for (int q = 0; q < Q; ++q)
            if (valid(q))
#pragma unroll
                for (int d = 0; d < 3; ++d) vec[3 * bead(q) + d] = x[q][d];
    }

    // Lanczos start vector (src/hydrodynamics.cpp:152-155): the warm-start
    // vector, normalised unless it is a unit vector to rounding (as every vector
    // of an earlier step is: a run then does not depend on where it was cut),
    // or the normalised default seed when cold or zero.
    __device__ void start_vector(bool warm, const double* cache, double (&v)[Q][3]) {
        if (warm) {
            load(cache, v);
            const double n2 = dot(v, v);
            if (n2 > 0.0) {
                if (fabs(n2 - 1.0) > 1.0e-13) {
                    const double inv = 1.0 / sqrt(n2);
#pragma unroll
                    for (int q = 0; q < Q; ++q)
#pragma unroll
                        for (int d = 0; d < 3; ++d) v[q][d] *= inv;
                }
                return;
            }
        }
        load(S.seed, v);
    }

    // w -= sum_i (V_i.w) V_i over the first nv vectors of the cold basis, all
    // projections reduced together (one barrier).
    __device__ __forceinline__ void project(int nv, double (&w)[Q][3]) {
        double* r = S.proj;
        sync();
#pragma unroll 1
        for (int u0 = 0; u0 < nv; u0 += 8) {
            double c[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                double x[Q][3], t = 0.0;
                load(Vg + (int64_t)min(u0 + i, nv - 1) * nv_stride(), x);
#pragma unroll
                for (int q = 0; q < Q; ++q)
#pragma unroll
                    for (int d = 0; d < 3; ++d) t += w[q][d] * x[q][d];
                c[i] = u0 + i < nv ? t : 0.0;
            }
            warp_sum8(c, r + u0 * T);
        }
        sync();
#pragma unroll 1
        for (int u = 0; u < nv; ++u) {
            double x[Q][3];
            load(Vg + (int64_t)u * nv_stride(), x);
            const double c = total(r, u);
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int d = 0; d < 3; ++d) w[q][d] -= c * x[q][d];
        }
    }
    __device__ __forceinline__ int nv_stride() const { return nv; }

    // Returns the number of Lanczos steps; sets rmin/rmax and the Ritz vectors.
    // v0: the start vector; if have_dv0, dv0 = D v0 (computed by the caller
    // together with the step's other independent products).
    // Warm runs (8 steps from the previous step's Ritz vectors) use the
    // three-term recurrence without reorthogonalisation: in 8 FP64 steps the
    // loss of orthogonality leaves the extreme Ritz values far inside the 2x /
    // 2% padding of the bounds, and the Chebyshev fluctuation-dissipation check
    // polices the result. Cold runs (30 steps, the first step of a call) project
    // on the whole basis where BasisLoss says so (below 3N = 64 in every step),
    // which keeps it orthogonal to the square root of the FP32 products' rounding;
    // the reference's modified Gram-Schmidt took up to 30 reductions in turn per
    // step. One reduction per
    // step: the new vector u goes into the product unnormalised, and u.u and u.Du
    // are summed together.
    __device__ int lanczos(int m, bool warm, const double (&v0)[Q][3], const double (&dv0)[Q][3], bool have_dv0,
                           double (&vmin)[Q][3], double (&vmax)[Q][3], double& rmin, double& rmax) {
        if (n < m) m = n;
        const bool cold = !(m <= kLanczosWarm), every = n < 64;
        double u[Q][3], w[Q][3], vp[Q][3];
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                u[q][d] = v0[q][d];
                w[q][d] = dv0[q][d];
                vp[q][d] = 0.0;
            }
        int k = 0;
        BasisLoss loss;
#pragma unroll 1
        for (int j = 0;; ++j) {
            if (j > 0 || !have_dv0) apply(u, w);
            double g[2] = {0.0, 0.0}, ww = 0.0;
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    g[0] += u[q][d] * u[q][d];
                    g[1] += u[q][d] * w[q][d];
                    ww += w[q][d] * w[q][d];
                }
            if (cold) {
                double g3[3] = {g[0], g[1], ww};
                sums(g3);
                g[0] = g3[0];
                g[1] = g3[1];
                ww = g3[2];
            } else {
                sums(g);
            }
            if (j > 0 && g[0] < 1.0e-20) {
                cnt[C_DX] -= 1;  // (the reference stops before this product)
                break;
            }
            const double ib = rsqrt_refined(g[0]), bt = g[0] * ib, al = (g[1] * ib) * ib;
            if (tid == 0) {
                S.alpha[j] = al;
                if (j > 0) S.beta[j - 1] = bt;
            }
            ++k;
            double v[Q][3];
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int d = 0; d < 3; ++d) v[q][d] = u[q][d] * ib;
            store(basis(j, m), v);
            if (j == m - 1) break;  // (the last beta is no entry of the tridiagonal)
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    u[q][d] = w[q][d] * ib - al * v[q][d];
                    if (j > 0) u[q][d] -= bt * vp[q][d];
                    vp[q][d] = v[q][d];
                }
            if (cold && (every || loss.project(j, al, bt, (ww * ib) * ib, 1.0e-7f, 3.0e-4f, 1.0e-5f))) project(j + 1, u);
        }
        sync();
        if (k == 1) {
            rmin = rmax = S.alpha[0];
            load(basis(0, m), vmin);
            load(basis(0, m), vmax);
            return 1;
        }
        if (wi == 0 && k <= kLanczosWarm) {
            // warm-sized tridiagonal in registers: Gershgorin bracket, then
            // lanes 0-15 find the smallest eigenvalue and its Ritz vector,
            // lanes 16-31 the largest
            double ar[kLanczosWarm], br[kLanczosWarm], b2[kLanczosWarm];
#pragma unroll
            for (int i = 0; i < kLanczosWarm; ++i) {
                ar[i] = i < k ? S.alpha[i] : 0.0;
                br[i] = i < k - 1 ? S.beta[i] : 0.0;
                b2[i] = br[i] * br[i];
            }
            double lo = ar[0], hi2 = ar[0];
#pragma unroll
            for (int i = 0; i < kLanczosWarm; ++i) {
                if (i < k) {
                    const double rad = (i > 0 ? fabs(br[i - 1]) : 0.0) + fabs(br[i]);
                    lo = dmin_(lo, ar[i] - rad);
                    hi2 = dmax_(hi2, ar[i] + rad);
                }
            }
            halfwarp_multisect(ar, b2, k, wl < 16 ? 1 : k, lo, hi2);
            const double r = 0.5 * (lo + hi2);
            double y[kLanczosWarm];
            tridiag_vec_reg<1>(ar, br, k, r, y);
            if ((wl & 15) == 0) {
                double* dst = wl == 0 ? S.ymin : S.ymax;
#pragma unroll
                for (int i = 0; i < kLanczosWarm; ++i)
                    if (i < k) dst[i] = y[i];
                S.rr[wl >> 4] = r;
            }
        } else if (wi == 0) {
            double lo = S.alpha[0], hi2 = S.alpha[0];
            for (int i = 0; i < k; ++i) {
                const double rad = (i > 0 ? fabs(S.beta[i - 1]) : 0.0) + (i < k - 1 ? fabs(S.beta[i]) : 0.0);
                lo = dmin_(lo, S.alpha[i] - rad);
                hi2 = dmax_(hi2, S.alpha[i] + rad);
            }
            // lanes 0-15 of the first warp bracket the smallest eigenvalue,
            // lanes 16-31 the largest
            double l2 = lo, h2 = hi2;
            halfwarp_bisect(S.alpha, S.beta, k, wl < 16 ? 1 : k, l2, h2);
            const double r = 0.5 * (l2 + h2);
            const double r0 = __shfl_sync(kFull, r, 0);
            const double r1 = __shfl_sync(kFull, r, 16);
            if (wl == 0 || wl == 16) {
                const bool lo_end = wl == 0;
                wk_tridiag_vec(S.alpha, S.beta, k, lo_end ? r0 : r1, lo_end ? S.ymin : S.ymax,
                               lo_end ? S.s3 : S.s3 + 32, lo_end ? S.s4 : S.s4 + 32);
            }
            if (wl == 0) {
                S.rr[0] = r0;
                S.rr[1] = r1;
            }
        }
        sync();
        rmin = S.rr[0];
        rmax = S.rr[1];
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
            for (int d = 0; d < 3; ++d) vmin[q][d] = vmax[q][d] = 0.0;
        for (int j = 0; j < k; ++j) {
            double vj[Q][3];
            load(basis(j, m), vj);
            const double y1 = S.ymin[j], y2 = S.ymax[j];
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    vmin[q][d] += y1 * vj[q][d];
                    vmax[q][d] += y2 * vj[q][d];
                }
        }
        sync();
        return k;
    }

    // spectral_bounds (src/hydrodynamics.cpp:224-264). v0: the start vector,
    // replaced by the next step's.
    // The step's three mutually independent products against D(R) run in
    // one pass first: D v0 (the Lanczos start vector), D X0 (the noise, for
    // the Chebyshev series) and D A (A = Fs + Fe, the predictor's force).
    // fuse: also form DX0 = D X0 and DA = D A in the start vector's pass;
    // otherwise the caller has them and the Lanczos forms D v0 itself.
    __device__ void bounds(double (&v0)[Q][3], int& cache_valid, double& lmin, double& lmax, const float (&X0)[Q][3],
                           const float (&A)[Q][3], float (&DX0)[Q][3], float (&DA)[Q][3], bool fuse = true) {
        double vmin[Q][3], vmax[Q][3], rmin, rmax;
        const bool can_warm = cache_valid != 0;
        double dv0[Q][3];
        if (fuse) {
            float x3[3][Q][3], y3[3][Q][3];
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    x3[0][q][d] = (float)v0[q][d];
                    x3[1][q][d] = X0[q][d];
                    x3[2][q][d] = A[q][d];
                }
            applyK<3>(x3, y3);
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    dv0[q][d] = (double)y3[0][q][d];
                    DX0[q][d] = y3[1][q][d];
                    DA[q][d] = y3[2][q][d];
                }
        }
        const int steps =
            lanczos(can_warm ? kLanczosWarm : kLanczosCold, can_warm, v0, dv0, fuse, vmin, vmax, rmin, rmax);
        if (can_warm && steps < 4) {
            start_vector(false, nullptr, v0);
            lanczos(kLanczosCold, false, v0, dv0, false, vmin, vmax, rmin, rmax);
            cnt[C_LZCOLD] += 1;
        } else {
            cnt[can_warm ? C_LZWARM : C_LZCOLD] += 1;
        }
        double sd[Q][3];
        load(S.seed, sd);
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
            for (int d = 0; d < 3; ++d) v0[q][d] = vmin[q][d] + vmax[q][d] + 0.01 * sd[q][d];
        const double s2 = dot(v0, v0);
        cache_valid = (s2 > 0.0 && isfinite(s2)) ? 1 : 0;
        const double is = rsqrt_refined(s2);
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
            for (int d = 0; d < 3; ++d) v0[q][d] = cache_valid ? v0[q][d] * is : sd[q][d];
        lmin = 0.5 * rmin;
        lmax = 1.02 * rmax;
        if (lmin < 1.0e-12) lmin = 1.0e-12;
        if (lmin >= lmax) lmin = lmax * 1.0e-6;
    }

    // ---- Chebyshev square root, FP32 recurrence (src/hydrodynamics.cpp:267-337)
    // Returns the FD error; out = approx D^{1/2} x0.
    // Dx0 = D x0 (computed by the caller). grow: the FD growth loop of the
    // reference; without it a failed check returns at once (bounds kept from
    // an earlier step are refreshed first).
    __device__ double chebyshev(const float (&x0)[Q][3], const float (&Dx0)[Q][3], double lmin, double lmax,
                                float (&out)[Q][3], bool grow = true) {
        const double x0Dx0 = dotf(x0, Dx0);
        double Lr = sqrt(lmax / lmin) * ch.mult + 0.5;
        int L = !(Lr < 2.0e9) ? kMaxCheb : (int)Lr + 1;
        L = L > kMaxCheb ? kMaxCheb : (L < 2 ? 2 : L);
        const float da = (float)(2.0 / (lmax - lmin));
        const float db = (float)(-(lmax + lmin) / (lmax - lmin));
        double fd = 0.0;
        for (;;) {
            // every cosine of the coefficient sums is cos(pi m / 2P), P = L + 1,
            // with integer m: one table of P + 1 values
            const int P = L + 1;
            const float ida = 1.f / da;
            for (int m = tid; m <= P; m += TT) ct[m] = cospif((float)m / (float)(2 * P));
            sync();
            for (int k = tid; k < P; k += TT) {
                const int m = 2 * k + 1;
                sqx[k] = sqrtf(((m <= P ? ct[m] : -ct[2 * P - m]) - db) * ida);
            }
            sync();
            for (int j = tid; j < P; j += TT) {
                float s = 0.f;
                int m = j;  // j (2k + 1) modulo 4P
                for (int k = 0; k < P; ++k) {
                    const int h = m > 2 * P ? 4 * P - m : m;
                    s += sqx[k] * (h <= P ? ct[h] : -ct[2 * P - h]);
                    m += 2 * j;
                    if (m >= 4 * P) m -= 4 * P;
                }
                s *= 2.f / (float)P;
                if (j == 0) s *= 0.5f;
                coef[j] = s;
            }
            sync();
            float tp[Q][3], tc[Q][3], o[Q][3];
            const float c0 = coef[0], c1 = coef[1];
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    tp[q][d] = x0[q][d];
                    tc[q][d] = da * Dx0[q][d] + db * tp[q][d];
                    o[q][d] = c0 * tp[q][d] + c1 * tc[q][d];
                }
            for (int l = 2; l <= L; ++l) {
                float Dv[Q][3];
                apply32(tc, Dv);
                const float cl = coef[l];
#pragma unroll
                for (int q = 0; q < Q; ++q)
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        const float tn = 2.f * (da * Dv[q][d] + db * tc[q][d]) - tp[q][d];
                        tp[q][d] = tc[q][d];
                        tc[q][d] = tn;
                        o[q][d] += cl * tn;
                    }
            }
            cnt[C_CHEB] += L;
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int d = 0; d < 3; ++d) out[q][d] = valid(q) ? o[q][d] : 0.f;
            const double rr = dotf(out, out);
            fd = fabs(rr - x0Dx0) / x0Dx0;
            sync();
            if (fd <= ch.fd_tol || L >= kMaxCheb || !grow) break;
            const int grow = L / 4 > 1 ? L / 4 : 1;
            L = (L + grow) > kMaxCheb ? kMaxCheb : L + grow;
        }
        return fd;
    }

    // ---- Cholesky fallback (src/mobility.cpp:69-81): dense FP64 D in global
    // scratch, right-looking factor, L x0. Returns false if not PD.
    __device__ bool cholesky_noise(const double (&R)[Q][3], const float (&x0)[Q][3], float (&out)[Q][3]) {
        to_smem(S.s0, R);
        sync();
        double* L = Lt;
        for (int idx = tid; idx < 9 * N; idx += TT) {
            const int mu = idx / 9, i = (idx % 9) / 3, j = idx % 3;
            L[(int64_t)(3 * mu + i) * n + 3 * mu + j] = (i == j) ? 1.0 : 0.0;
        }
        const int npairs = N * (N - 1) / 2;
        for (int pidx = tid; pidx < npairs; pidx += TT) {
            int nu = (int)((1.0 + sqrt(1.0 + 8.0 * (double)pidx)) * 0.5);
            while (nu * (nu - 1) / 2 > pidx) --nu;
            while ((nu + 1) * nu / 2 <= pidx) ++nu;
            const int mu = pidx - nu * (nu - 1) / 2;
            double b[3];
            for (int d = 0; d < 3; ++d) b[d] = S.s0[3 * nu + d] - S.s0[3 * mu + d];
            double om1, om2;
            rpy_weights(ch.hstar, b[0] * b[0] + b[1] * b[1] + b[2] * b[2], om1, om2);
            for (int i = 0; i < 3; ++i)
                for (int j = 0; j < 3; ++j) {
                    const double val = om2 * b[i] * b[j] + (i == j ? om1 : 0.0);
                    L[(int64_t)(3 * mu + i) * n + 3 * nu + j] = val;
                    L[(int64_t)(3 * nu + j) * n + 3 * mu + i] = val;
                }
        }
        __threadfence_block();
        sync();
        if (!team_factor<T>(L, n, tid, team)) return false;
#pragma unroll
        for (int q = 0; q < Q; ++q)
            if (valid(q))
#pragma unroll
                for (int d = 0; d < 3; ++d) S.s1[3 * bead(q) + d] = (double)x0[q][d];
        sync();
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const int i = 3 * bead(q) + d;
                double s = 0.0;
                if (valid(q))
                    for (int j = 0; j <= i; ++j) s += L[(int64_t)j * n + i] * S.s1[j];
                out[q][d] = (float)s;
            }
        sync();
        return true;
    }
};

// -------------------------------------------------------------- the kernel

template <int T, int Q>
__global__ void __launch_bounds__(TeamCfg<T, Q>::kCtaThreads, TeamCfg<T, Q>::kMinBlocks)
    integrate_team_kernel(const RunArgs a) {
    extern __shared__ __align__(16) unsigned char wsm[];
    constexpr int TT = TeamCfg<T, Q>::kThreads;
    const int team = threadIdx.x / TT;
    const int tid = threadIdx.x % TT;
    const int64_t stride = team_area_stride<T, Q>(a.n_max, a.w_pairs);
    TeamShared<T, Q>& S = *reinterpret_cast<TeamShared<T, Q>*>(wsm + stride * team);
    double* Vs = reinterpret_cast<double*>(wsm + stride * team + (sizeof(TeamShared<T, Q>) + 15) / 16 * 16);
    const int64_t gw = (int64_t)blockIdx.x * TeamCfg<T, Q>::kTeamsPerCta + team;
    double* scr = a.scratch + gw * a.scratch_stride;
    const int nvr = (int)round_up8(a.n_max);
    const uint64_t t_launch = global_ns();

    for (;;) {
        if (tid == 0) {
            const int item = atomicAdd(a.work_counter, 1);
            S.item = item >= a.n_work ? -1 : (a.order ? a.order[item] : item);
        }
        team_sync<T>(team);
        const int c = S.item;
        if (c < 0) break;
        {
            const int nw = (int)(sizeof(DevChain) / 8);
            const double* src = reinterpret_cast<const double*>(a.chains + c);
            double* dst = reinterpret_cast<double*>(&S.ch);
            for (int i = tid; i < nw; i += TT) dst[i] = src[i];
        }
        team_sync<T>(team);
        const DevChain& ch = S.ch;
        int status = a.status[c];
        if ((status & BDCU_ST_FATAL_MASK) || ch.bad_param) {
            if (tid == 0 && ch.bad_param) a.status[c] = status | BDCU_ST_BAD_PARAM;
            team_sync<T>(team);
            continue;
        }
        TeamChain<T, Q> W(a, S, ch);
        W.V = Vs;
        W.sqx = reinterpret_cast<float*>(Vs);
        W.coef = reinterpret_cast<float*>(Vs) + kCoefCap;
        W.ct = reinterpret_cast<float*>(Vs) + 2 * kCoefCap;
        W.Wt = reinterpret_cast<float4*>(reinterpret_cast<unsigned char*>(&S) + team_weight_offset<T, Q>(a.n_max));
        W.par = W.xpar = 0;
        W.Vg = scr;
        W.Lt = scr + (int64_t)kLanczosCold * nvr;
        W.nv = nvr;
        W.tid = tid;
        W.wl = tid & 31;
        W.wi = tid >> 5;
        W.team = team;
        W.N = ch.N;
        W.n = 3 * ch.N;
        W.jc = 4 * (int)min((int64_t)(ch.N + 3) / 4, a.w_pairs / (2 * ch.N));
        W.hi = ch.hstar > 0.0;
        W.status = status;
        for (int k = 0; k < 8; ++k) W.cnt[k] = 0;
        {
            const double RPI = 1.7724538509055160, TPI = 6.283185307179586;
            const double K1 = RPI * 0.75;
            W.scale = ch.hstar > 0.0 ? (float)ch.hstar : 1.f;
            W.iscale = 1.f / W.scale;
            W.K1 = (float)K1;
            W.K2 = (float)(K1 * (TPI / 3.0));
            W.K3 = (float)(K1 * TPI);
            W.C3 = (float)(0.75 / RPI * 0.375);
            W.C7 = (float)(0.09375 / RPI);
        }
        const int N = W.N;
        double* gR = a.R + 3 * ch.bead_off;
        double* gcache = a.cache + 3 * ch.bead_off;
        int cache_valid = (a.cache_mode == BDCU_CACHE_PERSIST) ? a.cache_valid[c] : 0;
        uint32_t ux = (uint32_t)a.rng[3 * c];
        int32_t iy = a.rng[3 * c + 1], sd = a.rng[3 * c + 2];
        W.noise_start(ux, iy, sd);
        bool drew = false, used_cache = false;
        double v0[Q][3];  // the Lanczos start vector, kept from step to step
        if (W.hi) {
            double s0[Q][3];
            W.load(a.seed_table, s0);
            const double iun = 1.0 / ch.seed_norm;
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int d = 0; d < 3; ++d) s0[q][d] *= iun;
            W.store(S.seed, s0);  // (each thread reads back only its own)
            W.start_vector(cache_valid != 0, gcache, v0);
        }
        double R[Q][3];
        W.load(gR, R);
        const int nsteps = a.n_steps[c];
        double t = a.t_start[c];
        const double dt = ch.dt;
        const double sqrt2inv = 1.0 / sqrt(2.0);
        const double sqrt_dt = sqrt(dt), inv_n = 1.0 / N;
        // spectral bounds kept between refreshes (a launch starts with a refresh)
        const int bounds_every = a.bounds_every > 1 ? a.bounds_every : 1;
        int since_bounds = bounds_every;
        double lmin = 0.0, lmax = 0.0;
        int step = 0;
        for (; step < nsteps; ++step) {
            // time slice: no new step past the budget (thread 0 decides for the team)
            if (a.budget_ns > 0 && W.tor(tid == 0 && (int64_t)(global_ns() - t_launch) >= a.budget_ns)) break;
            // recenter (src/integrator.cpp:88-93)
            if (ch.update_com) {
                double com[3];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    com[d] = 0.0;
#pragma unroll
                    for (int q = 0; q < Q; ++q) com[d] += R[q][d];
                }
                W.sums(com);
#pragma unroll
                for (int d = 0; d < 3; ++d) com[d] *= inv_n;
#pragma unroll
                for (int q = 0; q < Q; ++q)
                    if (W.valid(q))
                        for (int d = 0; d < 3; ++d) R[q][d] -= com[d];
            }
            W.stage_pos(R);
            float Fs[Q][3], Fe[Q][3];
            W.forces(R, t, Fs, Fe, true);
            float X0[Q][3], dW[Q][3], A[Q][3], DF[Q][3];
            W.noise(ux, iy, X0);
            drew = true;
            if (W.hi) W.build_weights();
            // brownian_step (src/mobility.cpp:58-88)
            if (!W.hi) {
#pragma unroll
                for (int q = 0; q < Q; ++q)
#pragma unroll
                    for (int d = 0; d < 3; ++d) dW[q][d] = (float)(sqrt_dt * X0[q][d]);
            } else {
                float bx[Q][3], DX0[Q][3];
#pragma unroll
                for (int q = 0; q < Q; ++q)
#pragma unroll
                    for (int d = 0; d < 3; ++d) A[q][d] = Fs[q][d] + Fe[q][d];
                double fd;
                if (since_bounds >= bounds_every) {
                    W.bounds(v0, cache_valid, lmin, lmax, X0, A, DX0, DF);
                    used_cache = true;
                    since_bounds = 0;
                    fd = W.chebyshev(X0, DX0, lmin, lmax, bx);
                } else {
                    // bounds kept from an earlier step: the two products in one pass
                    float x2[2][Q][3], y2[2][Q][3];
#pragma unroll
                    for (int q = 0; q < Q; ++q)
#pragma unroll
                        for (int d = 0; d < 3; ++d) {
                            x2[0][q][d] = X0[q][d];
                            x2[1][q][d] = A[q][d];
                        }
                    W.template applyK<2>(x2, y2);
#pragma unroll
                    for (int q = 0; q < Q; ++q)
#pragma unroll
                        for (int d = 0; d < 3; ++d) {
                            DX0[q][d] = y2[0][q][d];
                            DF[q][d] = y2[1][q][d];
                        }
                    fd = W.chebyshev(X0, DX0, lmin, lmax, bx, false);
                    if (!(fd <= ch.fd_tol)) {  // the kept bounds no longer hold: refresh and redo
                        W.bounds(v0, cache_valid, lmin, lmax, X0, A, DX0, DF, false);
                        used_cache = true;
                        since_bounds = 0;
                        fd = W.chebyshev(X0, DX0, lmin, lmax, bx);
                    }
                }
                ++since_bounds;
                if (!(fd <= ch.fd_tol)) {
                    W.status |= BDCU_ST_CHEB_FALLBACK;
                    W.cnt[C_FALLBACK] += 1;
                    if (!W.cholesky_noise(R, X0, bx)) {
                        W.status |= BDCU_ST_NOT_PD;
                        break;
                    }
                }
#pragma unroll
                for (int q = 0; q < Q; ++q)
#pragma unroll
                    for (int d = 0; d < 3; ++d) dW[q][d] = (float)(sqrt_dt * bx[q][d]);
            }
            // predictor (src/integrator.cpp:96-101)
            double K1[9], K2[9];
            kappa_at(ch, a.arena, t, K1);
            kappa_at(ch, a.arena, t + dt, K2);
            double Rp[Q][3];
            if (!W.hi)  // without HI D = I; with HI, bounds() formed D (Fs + Fe)
#pragma unroll
                for (int q = 0; q < Q; ++q)
#pragma unroll
                    for (int d = 0; d < 3; ++d) DF[q][d] = Fs[q][d] + Fe[q][d];
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int r = 0; r < 3; ++r) {
                    const double fl1 = K1[3 * r] * R[q][0] + K1[3 * r + 1] * R[q][1] + K1[3 * r + 2] * R[q][2];
                    Rp[q][r] = W.valid(q) ? R[q][r] + dt * (fl1 + 0.25 * DF[q][r]) + sqrt2inv * dW[q][r] : 0.0;
                }
            // upsilon (src/integrator.cpp:107-119): forces at R~ with R~'s coordinates staged
            W.stage_pos(Rp);
            float Fep[Q][3], dummy[Q][3];
            W.forces(Rp, t + dt, dummy, Fep, false);
            // D Fs + D (Fe + Fe~) = D (Fs + Fe) + D Fe~: the predictor's
            // product plus one more (the reference forms both sums anew)
            W.stage_pos(R);
            // solve_connectors (src/integrator.cpp:125-165): thread owns bonds
            // bead(0), bead(1). Its first iteration's bonds are those of R~,
            // so that iteration's product D Fb is formed in one pass with
            // upsilon's D Fe~.
            W.to_smem(S.s1, Rp);
            team_sync<T>(team);
            double bond[Q][3];
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const int b = W.bead(q);
#pragma unroll
                for (int d = 0; d < 3; ++d) bond[q][d] = b < N - 1 ? S.s1[3 * (b + 1) + d] - S.s1[3 * b + d] : 0.0;
            }
            const double anchor0 = S.s1[0], anchor1 = S.s1[1], anchor2 = S.s1[2];
            team_sync<T>(team);
            double Fc[Q][3];
            float Fb[Q][3], DFb[Q][3];
            // connector forces (src/spring.cpp:183-193) into s1, then the bead forces
            auto connector_and_bead_forces = [&]() {
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    const int b = W.bead(q);
                    const double f =
                        b < N - 1 ? connector_factor(ch, clamped_len(bond[q][0], bond[q][1], bond[q][2])) : 0.0;
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        Fc[q][d] = f * bond[q][d];
                        if (b < N - 1) S.s1[3 * b + d] = Fc[q][d];
                    }
                }
                team_sync<T>(team);
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    const int m = W.bead(q);
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        double v = 0.0;
                        if (m < N) {
                            if (m == 0) v = S.s1[d];
                            else if (m == N - 1) v = -S.s1[3 * (N - 2) + d];
                            else v = S.s1[3 * m + d] - S.s1[3 * (m - 1) + d];
                        }
                        Fb[q][d] = (float)v;
                    }
                }
                team_sync<T>(team);
            };
            connector_and_bead_forces();
            float DFep[Q][3];
            if (W.hi) {
                float x2[2][Q][3], y2[2][Q][3];
#pragma unroll
                for (int q = 0; q < Q; ++q)
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        x2[0][q][d] = Fep[q][d];
                        x2[1][q][d] = Fb[q][d];
                    }
                W.template applyK<2>(x2, y2);
#pragma unroll
                for (int q = 0; q < Q; ++q)
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        DFep[q][d] = y2[0][q][d];
                        DFb[q][d] = y2[1][q][d];
                    }
            } else {
#pragma unroll
                for (int q = 0; q < Q; ++q)
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        DFep[q][d] = Fep[q][d];
                        DFb[q][d] = Fb[q][d];
                    }
            }
            double ups[Q][3];
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int r = 0; r < 3; ++r) {
                    const double fl1 = K1[3 * r] * R[q][0] + K1[3 * r + 1] * R[q][1] + K1[3 * r + 2] * R[q][2];
                    const double fl2 = K2[3 * r] * Rp[q][0] + K2[3 * r + 1] * Rp[q][1] + K2[3 * r + 2] * Rp[q][2];
                    ups[q][r] = R[q][r] + dt * (0.5 * (fl1 + fl2) + 0.125 * ((double)DF[q][r] + (double)DFep[q][r])) +
                                sqrt2inv * dW[q][r];
                }
            W.to_smem(S.s0, ups);
            team_sync<T>(team);
            double dups[Q][3];
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const int b = W.bead(q);
#pragma unroll
                for (int d = 0; d < 3; ++d) dups[q][d] = b < N - 1 ? S.s0[3 * (b + 1) + d] - S.s0[3 * b + d] : 0.0;
            }
            team_sync<T>(team);
            double Rprev[Q][3], Rc[Q][3];
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int d = 0; d < 3; ++d) Rprev[q][d] = Rp[q][d];
            const int max_iter = 100 * N;
            const double c8 = 0.125 * dt, c4 = 0.25 * dt;
            int lstat = 0;
            for (int iter = 0;; ++iter) {
                if (iter > 0) {  // (the first iteration's Fc, Fb and D Fb are formed above)
                    connector_and_bead_forces();
                    W.applyF(Fb, DFb);
                }
#pragma unroll
                for (int q = 0; q < Q; ++q)
                    if (W.valid(q))
#pragma unroll
                        for (int d = 0; d < 3; ++d) S.s2[3 * W.bead(q) + d] = (double)DFb[q][d];
                team_sync<T>(team);
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    const int b = W.bead(q);
                    if (b < N - 1) {
                        double g[3], qv[3];
                        for (int d = 0; d < 3; ++d)
                            g[d] = dups[q][d] + c8 * (S.s2[3 * (b + 1) + d] - S.s2[3 * b + d]) + c4 * Fc[q][d];
                        solve_connector(g, dt, ch, qv, lstat);
                        for (int d = 0; d < 3; ++d) bond[q][d] = qv[d];
                    }
                }
                // R_corr = anchor + prefix sums of the bonds: inclusive scan in
                // each warp, then the totals of the warps before it (slot 0 of
                // the whole team precedes slot 1)
                double scan[Q][3];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    double v[Q];
#pragma unroll
                    for (int q = 0; q < Q; ++q) v[q] = bond[q][d];
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
                        for (int q = 0; q < Q; ++q) {
                            const double tq = __shfl_up_sync(kFull, v[q], o);
                            if (W.wl >= o) v[q] += tq;
                        }
                    }
#pragma unroll
                    for (int q = 0; q < Q; ++q) scan[q][d] = v[q];
                }
                if constexpr (T == 1) {
                    if constexpr (Q == 2) {
#pragma unroll
                        for (int d = 0; d < 3; ++d) scan[1][d] += __shfl_sync(kFull, scan[0][d], 31);
                    }
                    __syncwarp();
                } else {
                    if (W.wl == 31)
#pragma unroll
                        for (int q = 0; q < Q; ++q)
#pragma unroll
                            for (int d = 0; d < 3; ++d) S.tot[(q * 3 + d) * T + W.wi] = scan[q][d];
                    team_sync<T>(team);
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        double off0 = 0.0, all0 = 0.0, off1 = 0.0;
#pragma unroll
                        for (int w = 0; w < T; ++w) {
                            const double t0 = S.tot[d * T + w];
                            const double t1 = Q == 2 ? S.tot[(3 + d) * T + w] : 0.0;
                            if (w < W.wi) {
                                off0 += t0;
                                off1 += t1;
                            }
                            all0 += t0;
                        }
                        scan[0][d] += off0;
                        if constexpr (Q == 2) scan[1][d] += all0 + off1;
                    }
                }
                team_sync<T>(team);
                if (tid == 0) {
                    S.s1[0] = anchor0;
                    S.s1[1] = anchor1;
                    S.s1[2] = anchor2;
                }
                const double an[3] = {anchor0, anchor1, anchor2};
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    const int b = W.bead(q);
                    if (b < N - 1)
                        for (int d = 0; d < 3; ++d) S.s1[3 * (b + 1) + d] = an[d] + scan[q][d];
                }
                team_sync<T>(team);
                W.load(S.s1, Rc);
                team_sync<T>(team);
                double s = 0.0;
#pragma unroll
                for (int q = 0; q < Q; ++q)
                    if (W.valid(q)) {
                        const double e0 = Rc[q][0] - Rprev[q][0], e1 = Rc[q][1] - Rprev[q][1],
                                     e2 = Rc[q][2] - Rprev[q][2];
                        s += e0 * e0 + e1 * e1 + e2 * e2;
                    }
                const double incr = sqrt(W.tsum(s)) / N;
                W.cnt[C_CORR] += 1;
                if (incr < ch.tol) break;
                if (!(incr == incr) || isinf(incr)) {
                    W.status |= BDCU_ST_NONFINITE;
                    break;
                }
                if (iter >= max_iter) {
                    W.status |= BDCU_ST_NONCONVERGED;
                    W.cnt[C_NONCONV] += 1;
                    break;
                }
#pragma unroll
                for (int q = 0; q < Q; ++q)
#pragma unroll
                    for (int d = 0; d < 3; ++d) Rprev[q][d] = Rc[q][d];
            }
            // every thread's connector status, then a team-uniform fatal test
            W.status |= W.tor(lstat);
            if (W.status & BDCU_ST_FATAL_MASK) break;
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int d = 0; d < 3; ++d) R[q][d] = Rc[q][d];
            W.cnt[C_STEPS] += 1;
            t += dt;
        }
        if (used_cache && cache_valid) W.store(gcache, v0);
        if (!(W.status & BDCU_ST_FATAL_MASK)) W.store(gR, R);
        if (tid == 0) {
            if (drew) {  // (lazy seeding belongs to the first draw)
                a.rng[3 * c] = (int32_t)ux;
                a.rng[3 * c + 1] = iy;
                a.rng[3 * c + 2] = sd;
            }
            a.cache_valid[c] = cache_valid;
            a.status[c] = W.status;
            int64_t* cc = reinterpret_cast<int64_t*>(a.counters + c);
            for (int k = 0; k < 8; ++k) cc[k] += (int64_t)W.cnt[k];
            if (a.steps_done) a.steps_done[c] = step;
            if (a.t_end) a.t_end[c] = t;
        }
        team_sync<T>(team);
    }
}

}  // namespace bdcu
