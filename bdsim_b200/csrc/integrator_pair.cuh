// integrator_pair.cuh -- the FP64 plain form with the RPY tensor kept as pair
// weights: D.x needs, per bead pair, the two scalars omega1 and omega2 and the
// bead separation, so a chain's tensor is 16 bytes per pair (40 KB at N = 50)
// instead of the dense 72 (180 KB), and stays in shared memory. One chain per
// thread block of T warps, S lanes per bead (a power of two): every lane of a
// bead holds its state in registers, takes one part of its partner beads in the
// pair loops, and gets the bead's sum by shuffles.
//
// Every quantity is FP64 and every stage is the reference's; sums run in tree
// or segment order and the pair products use fma, so results differ from the
// reference's by rounding only (this file is compiled with --fmad=false: the
// spring, bending and connector arithmetic rounds as the reference's). The
// Lanczos runs project on the whole basis where a bound on the loss of orthogonality
// asks for it, all projections of a step reduced together (the reference projects
// every vector).
//
// Reference: src/integrator.cpp:61-170 of the bdsim project and the physics it
// calls; each stage cites its reference function.
#pragma once

#include "integrator.cuh"
#include "integrator_team.cuh"
#include "pair_layout.h"

namespace bdcu {

// Bracket of the target-th eigenvalue boundary by a whole warp: 31 Sturm
// counts at evenly spaced points per round, a ballot keeps one of the 32
// parts (five halvings of src/hydrodynamics.cpp:196-207 per round), until the
// interval is at rounding level.
template <typename Count>
__device__ __forceinline__ void warp_multisect(const Count& count, int target, double& lo, double& hi) {
    const int h = threadIdx.x & 31;
    for (int it = 0; it < 20; ++it) {
        const double w = hi - lo;
        const bool ge = h < 31 && count(fma(w, (double)(h + 1) * 0.03125, lo)) >= target;
        const unsigned bal = __ballot_sync(kFull, ge);
        const int f = bal ? __ffs(bal) - 1 : 31;
        const double nlo = f == 0 ? lo : fma(w, (double)f * 0.03125, lo);
        const double nhi = f == 31 ? hi : fma(w, (double)(f + 1) * 0.03125, lo);
        const bool done = (nlo == lo && nhi == hi) || (nhi - nlo) <= 2.5e-16 * fmax(fabs(nlo), fabs(nhi));
        lo = nlo;
        hi = nhi;
        if (done) break;
    }
}

// Beads are staged in pairs, components outermost within a pair: component d of
// bead j of one staged vector. The pair loops then read both beads of a pair
// with 16-byte loads at fixed offsets from one pointer.
__device__ __forceinline__ int pair_at(int j, int d) { return 6 * (j >> 1) + 2 * d + (j & 1); }

// Cholesky fallback (src/mobility.cpp:69-81), in four parts: the lower part of the
// dense D in global scratch from the staged positions ps (element (i, k) at L[k n +
// i]); its right-looking factor, eight columns at a time factored in shared memory
// (P, 8 round_up8(n) doubles: the area of the Chebyshev tables, dead by now) and
// taken off the trailing triangle, four of its columns per warp at once, so that an
// element crosses L2 once per eight columns and a lane's four loads are in flight
// together; y = L x (3N vectors in shared memory). Every element receives its
// products one by one, in k order. 148 chains of N = 50, 300 and 500, one step that
// falls back after 500 products: one column at a time 2.7, 170 and 712 ms, so 1.2, 39
// and 108. (The block kernel's tile updates on the tensor cores in this place: 32 and
// 70 ms for the long ones.) Each part out of line, with plain arguments and few
// registers: as one function, or with the tensor cores, it made the kernel spill in
// the steps that do not fall back (3 to 10% of long chains' time).
static __device__ __noinline__ void pair_dense(double* L, const double* ps, int N, double hstar) {
    const int n = 3 * N;
    for (int mu = threadIdx.x >> 5; mu < N; mu += blockDim.x >> 5)
        for (int nu = mu + (threadIdx.x & 31); nu < N; nu += 32) {
            double d[3], om1 = 1.0, om2 = 0.0;
            for (int k = 0; k < 3; ++k) d[k] = ps[pair_at(nu, k)] - ps[pair_at(mu, k)];
            if (mu != nu) rpy_weights(hstar, d[0] * d[0] + d[1] * d[1] + d[2] * d[2], om1, om2);
            double* col = L + (int64_t)(3 * mu) * n + 3 * nu;
            for (int j = 0; j < 3; ++j)
                for (int i = 0; i < 3; ++i) col[(int64_t)j * n + i] = om2 * d[i] * d[j] + (i == j ? om1 : 0.0);
        }
    __syncthreads();
}
constexpr int kPairPanel = 8;
// Columns k0 .. k0 + 7 (fewer at the end) into P, factored, and back. False if not
// positive definite.
static __device__ __noinline__ bool pair_panel(double* L, double* P, int n, int k0) {
    const int tid = threadIdx.x, TT = blockDim.x, ld = (n + 7) & ~7, kb = min(kPairPanel, n - k0);
    for (int u = 0; u < kb; ++u)
        for (int i = k0 + u + tid; i < n; i += TT) P[u * ld + i] = L[(int64_t)(k0 + u) * n + i];
    __syncthreads();
    for (int u = 0; u < kb; ++u) {
        const double s = P[u * ld + k0 + u];
        if (!(s > 0.0)) return false;
        const double dk = sqrt(s);
        __syncthreads();
        if (tid == 0) P[u * ld + k0 + u] = dk;
        for (int i = k0 + u + 1 + tid; i < n; i += TT) P[u * ld + i] = P[u * ld + i] / dk;
        __syncthreads();
        for (int v = u + 1; v < kb; ++v) {
            const double l = P[u * ld + k0 + v];
            for (int i = k0 + v + tid; i < n; i += TT) P[v * ld + i] -= P[u * ld + i] * l;
        }
        __syncthreads();
    }
    for (int u = 0; u < kb; ++u)
        for (int i = k0 + u + tid; i < n; i += TT) L[(int64_t)(k0 + u) * n + i] = P[u * ld + i];
    return true;
}
// The panel P of the eight columns before k1 off the columns from k1 on.
static __device__ __noinline__ void pair_trailing(double* L, const double* P, int n, int k1) {
    constexpr int kCols = 4;
    const int ld = (n + 7) & ~7;
    for (int j = k1 + kCols * (threadIdx.x >> 5); j < n; j += kCols * (blockDim.x >> 5)) {
        double* col = L + (int64_t)j * n;
#pragma unroll 1
        for (int i = j + (threadIdx.x & 31); i < n; i += 32) {
            double v[kCols];
#pragma unroll
            for (int c = 0; c < kCols; ++c) v[c] = i >= j + c ? col[(int64_t)c * n + i] : 0.0;
#pragma unroll 1
            for (int u = 0; u < kPairPanel; ++u) {
                const double f = P[u * ld + i];
#pragma unroll
                for (int c = 0; c < kCols; ++c) v[c] -= f * P[u * ld + min(j + c, n - 1)];
            }
#pragma unroll
            for (int c = 0; c < kCols; ++c)
                if (i >= j + c) col[(int64_t)c * n + i] = v[c];
        }
    }
    __syncthreads();
}
static __device__ __noinline__ void pair_lower(const double* L, int n, const double* x, double* y) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        double s = 0.0;
        for (int j = 0; j <= i; ++j) s += L[(int64_t)j * n + i] * x[j];
        y[i] = s;
    }
    __syncthreads();
}

// Doubles of a chain's factor in shared memory: its 3x3 blocks of the lower
// triangle, column by column.
__device__ __forceinline__ int factor_block(int N, int I, int J) { return 9 * (J * N - J * (J - 1) / 2 + (I - J)); }

template <int T>
struct PairChain {
    static constexpr int TT = 32 * T;
    const RunArgs& a;
    const DevChain& ch;
    double *red, *alpha, *beta, *ymin, *ymax, *tot, *ps, *pq, *xs, *buf, *s3, *s4, *area, *seed;
    double2* Wt;          // cached weights: (omega1, omega2) of this thread's e-th pair at Wt[e * S * Ne + wslot]
    int32_t* ctl;
    uint32_t* jcols;      // columns of the xorshift matrix power 3N
    double *Vg, *Lt;      // global: cold Lanczos basis, fallback factor (n x n)
    int ldv;
    int tid, wl, wi;
    int N, n, Ne;         // beads, 3N, N rounded up to even
    int S, seg, b, bc;    // lanes per bead, this lane's part, its bead (clamped to the chain: bc)
    int G;                // groups per warp: 2S lanes share two adjacent beads in D.x
    int gl, wslot;        // this lane's part in its group (lane / G), its column of the cached weights
    int np, nc;           // this lane's partner bead pairs 2 (gl + 2S i), +1, and how many have cached weights
    int par, xpar;        // parity of the reduction buffer and of the single products' input rows
    bool on, own, lane_on, hi;  // holds a bead; as its first lane; takes part in D.x; HI on
    RpyConst rpy;
    int32_t cnt[8];
    int status;

    __device__ PairChain(const RunArgs& a_, const DevChain& ch_) : a(a_), ch(ch_) {}

    // Neighbour-exchange buffers, 3N doubles each: 0 connector forces, 1 unit
    // bonds, then D Fb, 2 uniforms, then upsilon. Between a buffer's last read and
    // its next write there is always a barrier.
    __device__ __forceinline__ double* sb(int k) const { return buf + 3 * k * N; }

    // Sum over the S lanes of a bead, the same bits in each.
    __device__ __forceinline__ double bead_sum(double v) const {
        for (int o = 8; o >= G; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
        return v;
    }

    // Sums over the beads, the same bits in every thread: a butterfly over the
    // beads of each warp, then the T warps' sums in order (warps without beads
    // add zeros). One barrier: consecutive calls alternate between two buffers
    // of 32 values x T warps.
    __device__ __forceinline__ double* next_red() {
        double* r = red + par * (32 * T);
        par ^= 1;
        return r;
    }
    template <int M>
    __device__ __forceinline__ void sums(double (&v)[M]) {
        double* r = next_red();
#pragma unroll
        for (int m = 0; m < M; ++m) v[m] += __shfl_xor_sync(kFull, v[m], 16);
#pragma unroll 1
        for (int o = 1; o < G; o <<= 1)
#pragma unroll
            for (int m = 0; m < M; ++m) v[m] += __shfl_xor_sync(kFull, v[m], o);
        if (wl == 0)
#pragma unroll
            for (int m = 0; m < M; ++m) r[m * T + wi] = v[m];
        __syncthreads();
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const double2* q = reinterpret_cast<const double2*>(r + m * T);
            double a0 = T == 1 ? 0.0 + r[m] : 0.0;
#pragma unroll
            for (int w = 0; w < T / 2; ++w) a0 += q[w].x + q[w].y;
            v[m] = a0;
        }
    }
    // After a barrier: lane l gets the total over the warps of value l & 7 of
    // the eight published at r (one load per four warps, two shuffles).
    __device__ __forceinline__ double total8(const double* r) const {
        const double* q = r + (wl & 7) * T + (wl >> 3);
        double t = T >= 4 || (wl >> 3) < T ? q[0] : 0.0;
#pragma unroll
        for (int w = 4; w < T; w += 4) t += q[w];
        t += __shfl_xor_sync(kFull, t, 8);
        t += __shfl_xor_sync(kFull, t, 16);
        return t;
    }
    __device__ __forceinline__ double dot(const double (&x)[3], const double (&y)[3]) {
        double v[1] = {fma(x[2], y[2], fma(x[1], y[1], x[0] * y[0]))};
        sums(v);
        return v[0];
    }
    __device__ __forceinline__ int any_bits(int v) {
        if (tid == 0) ctl[0] = 0;
        __syncthreads();
        v = __reduce_or_sync(kFull, v);
        if (wl == 0 && v) atomicOr(ctl, v);
        __syncthreads();
        return ctl[0];
    }

    // ---- D.x ------------------------------------------------------------
    // K products at once: x[r] at the thread's bead, y[r] = (D x[r]) there. Per
    // pair: the separation (3 adds), d.x (3), omega2 d.x (1) and six fma,
    // against two cached doubles (a 16-byte load of the thread's own), or
    // against weights evaluated here (~20 more operations) beyond the cached
    // ones. The 2S lanes of two adjacent beads share their work: each takes
    // both beads against every 2S-th pair of partner beads, so that the partner
    // loads (16-byte broadcasts, two shared-memory cycles each) serve two
    // beads: one bead per lane is bound by those loads (1080 cycles per product
    // and SM at N = 50, against 740 for the arithmetic). One barrier:
    // consecutive single products alternate between input rows, and every other
    // reuse of the rows lies behind a reduction's barrier.
    template <int K>
    __device__ __forceinline__ void apply(const double (&x)[K][3], double (&y)[K][3]) {
        if (!hi) {
#pragma unroll
            for (int r = 0; r < K; ++r)
#pragma unroll
                for (int d = 0; d < 3; ++d) y[r][d] = x[r][d];
            return;
        }
        cnt[C_DX] += K;
        double* xr = xs;
        if (K == 1) {
            xr += xpar * 3 * Ne;
            xpar ^= 1;
        }
        if (own)
#pragma unroll
            for (int r = 0; r < K; ++r)
#pragma unroll
                for (int d = 0; d < 3; ++d) xr[6 * K * (b >> 1) + 6 * r + 2 * d + (b & 1)] = x[r][d];
        if ((N & 1) && tid < 3 * K) xr[6 * K * (N >> 1) + 2 * tid + 1] = 0.0;
        __syncthreads();
        double acc[K][2][3];
#pragma unroll
        for (int r = 0; r < K; ++r)
#pragma unroll
            for (int d = 0; d < 3; ++d) acc[r][0][d] = acc[r][1][d] = 0.0;
        if (lane_on) {
            double q[2][3];
            group_beads(ps, q);
            const double2* pp = reinterpret_cast<const double2*>(ps) + 3 * gl;
            const double2* xp = reinterpret_cast<const double2*>(xr) + 3 * K * gl;
            auto pairs = [&](const double2 (&wt)[2][2], const double2 (&p)[3]) {
                double dd[2][2][3];
#pragma unroll
                for (int e = 0; e < 2; ++e)
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        dd[e][0][d] = p[d].x - q[e][d];
                        dd[e][1][d] = p[d].y - q[e][d];
                    }
#pragma unroll
                for (int r = 0; r < K; ++r) {
                    const double2 u0 = xp[3 * r], u1 = xp[3 * r + 1], u2 = xp[3 * r + 2];
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const double(&da)[3] = dd[e][0];
                        const double(&db)[3] = dd[e][1];
                        const double2 wa = wt[e][0], wb = wt[e][1];
                        const double ta = wa.y * fma(da[2], u2.x, fma(da[1], u1.x, da[0] * u0.x));
                        const double tb = wb.y * fma(db[2], u2.y, fma(db[1], u1.y, db[0] * u0.y));
                        double(&y)[3] = acc[r][e];
                        y[0] = fma(tb, db[0], fma(wb.x, u0.y, fma(ta, da[0], fma(wa.x, u0.x, y[0]))));
                        y[1] = fma(tb, db[1], fma(wb.x, u1.y, fma(ta, da[1], fma(wa.x, u1.x, y[1]))));
                        y[2] = fma(tb, db[2], fma(wb.x, u2.y, fma(ta, da[2], fma(wa.x, u2.x, y[2]))));
                    }
                }
            };
            const double2* w = Wt + wslot;
            const int ws = S * Ne, dp = 6 * S;
            int i = 0;
            if (nc > 0) {  // the next step's weights and positions are loaded before this one's arithmetic
                double2 wt[2][2] = {{w[0], w[ws]}, {w[2 * ws], w[3 * ws]}}, p[3] = {pp[0], pp[1], pp[2]};
#pragma unroll 1
                for (;; xp += K * dp) {
                    const bool more = ++i < nc;
                    if (more) {
                        w += 4 * ws;
                        pp += dp;
                    }
                    const double2 wn[2][2] = {{w[0], w[ws]}, {w[2 * ws], w[3 * ws]}}, pn[3] = {pp[0], pp[1], pp[2]};
                    pairs(wt, p);
                    if (!more) break;
#pragma unroll
                    for (int e = 0; e < 2; ++e) wt[e][0] = wn[e][0], wt[e][1] = wn[e][1];
#pragma unroll
                    for (int d = 0; d < 3; ++d) p[d] = pn[d];
                }
                pp += dp;
                xp += K * dp;
            }
#pragma unroll 1
            for (; i < np; ++i, pp += dp, xp += K * dp) {
                const double2 p[3] = {pp[0], pp[1], pp[2]};
                double2 wt[2][2];
                weights4(2 * (gl + 2 * S * i), p, q, wt);
                pairs(wt, p);
            }
        }
        // each lane keeps its own bead's sums: halves of the group exchange,
        // then a butterfly over the bead's lanes
#pragma unroll
        for (int r = 0; r < K; ++r)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const bool up = wl >= 16;
                const double mine = up ? acc[r][1][d] : acc[r][0][d], other = up ? acc[r][0][d] : acc[r][1][d];
                const double v = bead_sum(mine + __shfl_xor_sync(kFull, other, 16));
                y[r][d] = on ? v : 0.0;
            }
    }
    __device__ __forceinline__ void apply1(const double (&x)[3], double (&y)[3]) {
        apply<1>(reinterpret_cast<const double(&)[1][3]>(x), reinterpret_cast<double(&)[1][3]>(y));
    }

    // The two beads of this thread's group at the staged positions p.
    __device__ __forceinline__ void group_beads(const double* p, double (&q)[2][3]) const {
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int d = 0; d < 3; ++d) q[e][d] = p[pair_at(b & ~1, d) + e];
    }

    // Weights of the group's two beads with beads j, j + 1 (positions p).
    __device__ __forceinline__ void weights4(int j, const double2 (&p)[3], const double (&q)[2][3],
                                             double2 (&wt)[2][2]) const {
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const double dx = (h ? p[0].y : p[0].x) - q[e][0], dy = (h ? p[1].y : p[1].x) - q[e][1],
                             dz = (h ? p[2].y : p[2].x) - q[e][2];
                rpy.weights(fma(dz, dz, fma(dy, dy, dx * dx)), j + h == (b & ~1) + e, wt[e][h].x, wt[e][h].y);
            }
    }

    // Weights of this thread's pairs at the staged positions (each thread reads
    // back only what it wrote: no barrier). The pad bead of an odd N meets zero
    // inputs only, and its sums are dropped.
    __device__ __forceinline__ void build_weights() {
        if (!lane_on) return;
        double q[2][3];
        group_beads(ps, q);
        const double2* pp = reinterpret_cast<const double2*>(ps) + 3 * gl;
        const int ws = S * Ne;
        double2* w = Wt + wslot;
#pragma unroll 1
        for (int i = 0; i < nc; ++i, pp += 6 * S, w += 4 * ws) {
            const double2 p[3] = {pp[0], pp[1], pp[2]};
            double2 wt[2][2];
            weights4(2 * (gl + 2 * S * i), p, q, wt);
            w[0] = wt[0][0];
            w[ws] = wt[0][1];
            w[2 * ws] = wt[1][0];
            w[3 * ws] = wt[1][1];
        }
    }

    __device__ __forceinline__ void stage(double* p, const double (&R)[3]) const {
        if (own)
#pragma unroll
            for (int d = 0; d < 3; ++d) p[pair_at(b, d)] = R[d];
        if ((N & 1) && tid < 3) p[pair_at(N, tid)] = 0.0;
        __syncthreads();
    }

    // ---- forces at the staged positions p -----------------------------------
    // Fs: spring bead forces (src/spring.cpp:195-207). Fe: (EV + bending) +
    // external(t) (src/model.hpp:56-64).
    __device__ __forceinline__ void forces(const double* p, double t, double (&Fs)[3], double (&Fe)[3], bool spring) {
        double f[3] = {0.0, 0.0, 0.0};
        if (ch.ev_type != BDCU_EV_NONE) {
            if (on) ev_part(p, f);
#pragma unroll
            for (int d = 0; d < 3; ++d) f[d] = bead_sum(f[d]);
        }
        const bool bend = ch.bend_type != BDCU_BEND_NONE && N > 2;
        double* Fc = sb(0);
        double* u = sb(1);
        if (spring || bend) {
            if (own && b < N - 1) {
                const int e0 = pair_at(b, 0), e1 = pair_at(b + 1, 0);
                const double b0 = p[e1] - p[e0], b1 = p[e1 + 2] - p[e0 + 2], b2 = p[e1 + 4] - p[e0 + 4];
                const double len = clamped_len(b0, b1, b2);
                if (spring) {
                    const double g = connector_factor(ch, len);
                    Fc[3 * b] = g * b0;
                    Fc[3 * b + 1] = g * b1;
                    Fc[3 * b + 2] = g * b2;
                }
                if (bend) {
                    const double il = 1.0 / len;
                    u[3 * b] = il * b0;
                    u[3 * b + 1] = il * b1;
                    u[3 * b + 2] = il * b2;
                    s3[b] = len;
                }
            }
            __syncthreads();
            if (bend) {
                if (own && b < N - 2)
                    s4[b] = u[3 * (b + 1)] * u[3 * b] + u[3 * (b + 1) + 1] * u[3 * b + 1] +
                            u[3 * (b + 1) + 2] * u[3 * b + 2];
                __syncthreads();
            }
        }
        for (int d = 0; d < 3; ++d) Fs[d] = Fe[d] = 0.0;
        if (on) {
            if (spring) bead_force(Fc, Fs);
            double fb[3] = {0.0, 0.0, 0.0}, fx[3] = {0.0, 0.0, 0.0};
            if (bend) bending_on_bead(ch, b, u, s4, s3, fb);
            if (ch.ext_n > 0) external_on_bead(ch, a.arena, b, t, fx);
            for (int d = 0; d < 3; ++d) Fe[d] = (f[d] + fb[d]) + fx[d];
        }
    }
    __device__ __forceinline__ void bead_force(const double* Fc, double (&F)[3]) const {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            if (b == 0) F[d] = Fc[d];
            else if (b == N - 1) F[d] = -Fc[3 * (N - 2) + d];
            else F[d] = Fc[3 * b + d] - Fc[3 * (b - 1) + d];
        }
    }

    // Excluded-volume force on this bead from this lane's part of the beads
    // (ExcludedVolume::force, src/excluded_volume.cpp:60-89): the force from j
    // is -fac (R_j - R_b), contour distance at least cd.
    __device__ __forceinline__ void ev_part(const double* p, double (&f)[3]) const {
        const double qx = p[pair_at(b, 0)], qy = p[pair_at(b, 1)], qz = p[pair_at(b, 2)];
        const int cd = ch.cd > 1 ? ch.cd : 1;
        if (ch.ev_type == BDCU_EV_GAUSS) {
            const double zs = ch.zsbyds5, p5 = ch.pt5bydssq;
#pragma unroll 4
            for (int j = seg; j < N; j += S) {
                const double* pj = p + pair_at(j, 0);
                const double dx = pj[0] - qx, dy = pj[2] - qy, dz = pj[4] - qz;
                const double sq = fmax(fma(dz, dz, fma(dy, dy, dx * dx)), 1.0e-12);
                const int dj = j > b ? j - b : b - j;
                const double fac = (dj >= cd ? zs : 0.0) * exp(-(sq * p5));  // (no branch around the exponential)
                f[0] = fma(-fac, dx, f[0]);
                f[1] = fma(-fac, dy, f[1]);
                f[2] = fma(-fac, dz, f[2]);
            }
            return;
        }
        // LJ and SDK vanish beyond their outer cutoff; pairs well outside are
        // passed over on the squared distance (the cutoff itself is tested on r)
        const double cut = ev_outer_cutoff(ch), cut2 = cut * cut * (1.0 + 1e-9);
        const double* phi = (ch.ev_type == BDCU_EV_SDK && ch.phi_off >= 0) ? a.arena + ch.phi_off : nullptr;
#pragma unroll 2
        for (int j = seg; j < N; j += S) {
            const double* pj = p + pair_at(j, 0);
                const double dx = pj[0] - qx, dy = pj[2] - qy, dz = pj[4] - qz;
            const double sq = fmax(fma(dz, dz, fma(dy, dy, dx * dx)), 1.0e-12);
            const int dj = j > b ? j - b : b - j;
            if (dj < cd || sq > cut2) continue;
            const int mu = j < b ? j : b, nu = j < b ? b : j;
            const double fac = ev_factor_short(ch, sq, phi ? phi + (int64_t)mu * N + nu : nullptr);
            f[0] = fma(-fac, dx, f[0]);
            f[1] = fma(-fac, dy, f[1]);
            f[2] = fma(-fac, dz, f[2]);
        }
    }

    // ---- noise: the 3N draws of raw_noise (src/mobility.cpp:18-29) ----------
    // The threads draw contiguous blocks of c draws of the stream. Each keeps
    // the generator's state at the start of its block: jumped there once per
    // chain, and from step to step by the same 3N draws for every thread (the
    // xorshift matrix power's columns in shared memory; 16807^3N mod 2^31 - 1).
    // State (ux, iy) of the chain's stream -> this thread's block start.
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
        if (tid < 32) jcols[tid] = a.xs_pow[32 * (int64_t)n + tid];
        __syncthreads();
    }
    __device__ __forceinline__ void noise(uint32_t& ux0, int32_t& iy0, double (&X)[3]) {
        const int c = (n + TT - 1) / TT, k0 = tid * c, k1 = min(n, k0 + c);
        double* y = sb(2);
        const float am = __fdiv_rn(__int_as_float(0x3f7fffff), 2147483648.0f);
        uint32_t ux = ux0, iy = (uint32_t)iy0;
        for (int k = k0; k < k1; ++k) {
            ux ^= (ux << 13);
            ux ^= (ux >> 17);
            ux ^= (ux << 5);
            iy = lehmer_mul(16807u, iy);
            const int32_t res = (int32_t)(((ux ^ iy) & 0x7fffffffu) | 1u);
            y[k] = (double)__fmul_rn(am, __int2float_rn(res));
        }
        ux0 = xorshift_jump(jcols, ux0);
        iy0 = (int32_t)lehmer_mul(a.a_pow[n], (uint32_t)iy0);
        __syncthreads();
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            X[d] = 0.0;
            if (on) {
                const double v = y[3 * b + d] - 0.5;
                X[d] = (14.14855378 * v * v + 1.21569221) * v;
            }
        }
    }

    // ---- Cholesky method (brownian_step, src/mobility.cpp:58-88) for chains of
    // up to kPairCholMaxN beads: D at the staged positions, factored in shared
    // memory (F, in the weights' place) one bead at a time: the 3x3 diagonal
    // block by every thread for itself, the rows below it one per thread, then
    // the trailing blocks, one warp per block column (two barriers per bead;
    // the block kernel takes three per matrix column and one thread's work
    // between two of them). Each element receives its products in k order
    // before its division, as in the reference. y = L x. False if not positive
    // definite.
    __device__ __forceinline__ bool cholesky_noise(const double (&x0)[3], double (&out)[3]) {
        double* F = reinterpret_cast<double*>(Wt);
        for (int J = wi; J < N; J += T)
            for (int I = J + wl; I < N; I += 32) {
                double d[3], om1, om2;
#pragma unroll
                for (int k = 0; k < 3; ++k) d[k] = ps[pair_at(I, k)] - ps[pair_at(J, k)];
                rpy.weights(fma(d[2], d[2], fma(d[1], d[1], d[0] * d[0])), I == J, om1, om2);
                double* f = F + factor_block(N, I, J);
#pragma unroll
                for (int i = 0; i < 3; ++i)
#pragma unroll
                    for (int j = 0; j < 3; ++j) f[3 * i + j] = om2 * d[i] * d[j] + (i == j ? om1 : 0.0);
            }
        __syncthreads();
#pragma unroll 1
        for (int K = 0; K < N; ++K) {
            double* f = F + factor_block(N, K, K);
            double l[3][3], r[3];
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j <= i; ++j) l[i][j] = f[3 * i + j];
            bool pd = true;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const double s = l[k][k];
                pd = pd && s > 0.0;
                r[k] = s > 1.0e-30 ? rsqrt_refined(s) : 1.0 / sqrt(s);
                l[k][k] = s * r[k];
#pragma unroll
                for (int i = k + 1; i < 3; ++i) l[i][k] *= r[k];
#pragma unroll
                for (int i = k + 1; i < 3; ++i)
#pragma unroll
                    for (int j = k + 1; j <= i; ++j) l[i][j] = fma(-l[i][k], l[j][k], l[i][j]);
            }
            if (!pd) return false;  // (every thread found the same)
            for (int I = K + 1 + tid; I < N; I += TT) {
                double* g = F + factor_block(N, I, K);
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const double a0 = g[3 * i] * r[0], a1 = fma(-a0, l[1][0], g[3 * i + 1]) * r[1],
                                 a2 = fma(-a1, l[2][1], fma(-a0, l[2][0], g[3 * i + 2])) * r[2];
                    g[3 * i] = a0;
                    g[3 * i + 1] = a1;
                    g[3 * i + 2] = a2;
                }
            }
            __syncthreads();
            if (tid == 0)
#pragma unroll
                for (int i = 0; i < 3; ++i)
#pragma unroll
                    for (int j = 0; j < 3; ++j) f[3 * i + j] = j <= i ? l[i][j] : 0.0;
            for (int J = K + 1 + wi; J < N; J += T)
                for (int I = J + wl; I < N; I += 32) {
                    const double *p = F + factor_block(N, I, K), *q = F + factor_block(N, J, K);
                    double* c = F + factor_block(N, I, J);
#pragma unroll
                    for (int i = 0; i < 3; ++i)
#pragma unroll
                        for (int j = 0; j < 3; ++j)
                            c[3 * i + j] = fma(-p[3 * i + 2], q[3 * j + 2],
                                               fma(-p[3 * i + 1], q[3 * j + 1], fma(-p[3 * i], q[3 * j], c[3 * i + j])));
                }
            __syncthreads();
        }
        double* x = sb(0);
        if (own)
#pragma unroll
            for (int d = 0; d < 3; ++d) x[3 * b + d] = x0[d];
        __syncthreads();
#pragma unroll
        for (int d = 0; d < 3; ++d) out[d] = 0.0;
        if (on)  // the lanes of a bead share its row of blocks
            for (int J = seg; J <= b; J += S) {
                const double* f = F + factor_block(N, b, J);
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    out[d] += fma(f[3 * d + 2], x[3 * J + 2], fma(f[3 * d + 1], x[3 * J + 1], f[3 * d] * x[3 * J]));
            }
#pragma unroll
        for (int d = 0; d < 3; ++d) out[d] = bead_sum(out[d]);
        __syncthreads();  // (x and F are free again)
        return true;
    }

    // ---- Lanczos extreme eigenvalues (src/hydrodynamics.cpp:146-264) --------

    // The sums of c[0..7] over the warp's beads into out[u * T + warp]: halves of the
    // vector exchanged with lanes ^16, ^8, ^4 (lanes of one bead hold the same
    // values and only select), then a butterfly over ^2, ^1.
    __device__ __forceinline__ void warp_sum8(const double (&c)[8], double* out) const {
        const bool u16 = wl & 16, u8 = wl & 8, u4 = wl & 4;
        double k4[4], k2[2], s;
#pragma unroll
        for (int u = 0; u < 4; ++u)
            k4[u] = (u16 ? c[u + 4] : c[u]) + __shfl_xor_sync(kFull, u16 ? c[u] : c[u + 4], 16);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            k2[u] = u8 ? k4[u + 2] : k4[u];
            if (8 < G) k2[u] += __shfl_xor_sync(kFull, u8 ? k4[u] : k4[u + 2], 8);
        }
        s = u4 ? k2[1] : k2[0];
        if (4 < G) s += __shfl_xor_sync(kFull, u4 ? k2[0] : k2[1], 4);
        if (2 < G) s += __shfl_xor_sync(kFull, s, 2);
        if (1 < G) s += __shfl_xor_sync(kFull, s, 1);
        if ((wl & 3) == 0) out[(wl >> 2) * T + wi] = s;
    }

    // Lanczos start vector (src/hydrodynamics.cpp:152-155): the warm-start
    // vector, normalised unless it is a unit vector to rounding (as every vector
    // of an earlier step is: a run then does not depend on where it was cut),
    // or the normalised default seed when cold or zero.
    __device__ __forceinline__ bool start_vector(const double* cache, bool warm, double (&v)[3]) {
        for (int d = 0; d < 3; ++d) v[d] = 0.0;
        if (warm) {
            if (on)
                for (int d = 0; d < 3; ++d) v[d] = cache[3 * b + d];
            const double n2 = dot(v, v);
            if (n2 > 0.0) {
                if (fabs(n2 - 1.0) > 1.0e-13) {
                    const double nv = sqrt(n2);
                    for (int d = 0; d < 3; ++d) v[d] = v[d] / nv;
                }
                return true;
            }
        }
        if (on)
            for (int d = 0; d < 3; ++d) v[d] = seed[3 * b + d];
        return warm;
    }

    // u -= sum_i (V_i.u) V_i over the first nv vectors of the cold basis, all
    // projections reduced together (one barrier).
    __device__ __forceinline__ void project(int nv, double (&u)[3]) {
        double* r = next_red();
#pragma unroll 1
        for (int u0 = 0; u0 < nv; u0 += 8) {
            double c[8];  // (loads without a branch, so that they are all in flight together)
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const double* vi = Vg + min(u0 + i, nv - 1) * ldv + 3 * bc;
                const double x = fma(u[2], vi[2], fma(u[1], vi[1], u[0] * vi[0]));
                c[i] = u0 + i < nv && on ? x : 0.0;
            }
            warp_sum8(c, r + u0 * T);
        }
        __syncthreads();
#pragma unroll 1
        for (int u0 = 0; u0 < nv; u0 += 8) {
            const double t = total8(r + u0 * T);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const double g = __shfl_sync(kFull, t, i), c = u0 + i < nv ? g : 0.0;
                const double* vi = Vg + min(u0 + i, nv - 1) * ldv + 3 * bc;
#pragma unroll
                for (int d = 0; d < 3; ++d) u[d] = on ? fma(-c, vi[d], u[d]) : 0.0;
            }
        }
    }

    // A Lanczos run from the unit vector v (with w = D v if have_w): 8 steps
    // with the basis in shared memory (warm), or 30 with it in global scratch
    // (cold, the first step of a call). One reduction per step: the new vector u
    // goes into the product unnormalised, and u.u and u.Du are summed together,
    // so that its norm (explicit: |Du|^2 - alpha^2 - beta^2 loses digits from
    // step to step), alpha and the next vector follow at once.
    // Orthogonality: the reference projects every vector on the whole basis. In 8
    // steps the three-term recurrence alone gives the same extreme eigenvalues to
    // 1e-12 relative (3e-10 for the smallest one of chains whose beads nearly
    // coincide). A cold run projects where BasisLoss says so (from 3N = 64; in
    // every step below, where the Krylov space is soon exhausted), which keeps the
    // basis orthogonal to 1e-8, the square root of rounding that the tridiagonal's
    // accuracy needs (3e-10 at most on rods, rings, coils and collapsed chains). (Projecting in every step read the basis from
    // L2 twice a step: 12.9 thousand cycles a step at N = 50, 2.7 of them the
    // product.) Returns its steps; the tridiagonal is left in alpha and beta.
    __device__ __forceinline__ int lanczos(double* V, bool cold, double (&v)[3], double (&w)[3], bool have_w) {
        const int m = min(n, cold ? kLanczosCold : kLanczosWarm);
        const bool every = n < 64;
        double u[3] = {v[0], v[1], v[2]}, vp[3] = {0.0, 0.0, 0.0};
        BasisLoss loss;
#pragma unroll 1
        for (int j = 0;; ++j) {
            if (j > 0 || !have_w) apply1(u, w);
            double g2[2] = {fma(u[2], u[2], fma(u[1], u[1], u[0] * u[0])), fma(u[2], w[2], fma(u[1], w[1], u[0] * w[0]))};
            double ww = 0.0;
            if (cold) {
                double g3[3] = {g2[0], g2[1], fma(w[2], w[2], fma(w[1], w[1], w[0] * w[0]))};
                sums(g3);
                g2[0] = g3[0];
                g2[1] = g3[1];
                ww = g3[2];
            } else {
                sums(g2);
            }
            const double bsq = g2[0];
            if (j > 0 && bsq < 1.0e-20) {
                cnt[C_DX] -= 1;  // (the reference stops before this product)
                return j;
            }
            const double ib = rsqrt_refined(bsq), al = (g2[1] * ib) * ib, bt = bsq * ib;
            if (tid == 0) {
                alpha[j] = al;
                if (j > 0) beta[j - 1] = bt;
            }
#pragma unroll
            for (int d = 0; d < 3; ++d) v[d] = u[d] * ib;
            if (own)
#pragma unroll
                for (int d = 0; d < 3; ++d) V[j * ldv + 3 * b + d] = v[d];
            if (j == m - 1) return m;  // (the last beta is no entry of the tridiagonal)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                u[d] = fma(w[d], ib, -(al * v[d]));
                if (j > 0) u[d] = fma(-bt, vp[d], u[d]);
                vp[d] = v[d];
            }
            if (cold) {
                __syncwarp();  // (the lanes of a bead read its basis entries back)
                if (every || loss.project(j, al, bt, (ww * ib) * ib, 4.0e-16f, 1.0e-8f, 1.0e-10f)) project(j + 1, u);
            }
        }
    }

    // Extreme eigenvalues of the k x k tridiagonal and the sum of their two
    // Ritz vectors.
    __device__ __forceinline__ void ritz_pair(const double* V, int k, double (&ritz)[3], double& rmin, double& rmax) {
        __syncthreads();
        if (k == 1) {
            rmin = rmax = alpha[0];
            for (int d = 0; d < 3; ++d) ritz[d] = on ? 2.0 * V[3 * b + d] : 0.0;
            return;
        }
        for (int e = wi; e < 2; ++e) {  // warp 0 the smallest eigenvalue, warp 1 (or the only one) the largest
            double lo = alpha[0], hi2 = alpha[0];
            for (int i = 0; i < k; ++i) {
                const double rad = (i > 0 ? fabs(beta[i - 1]) : 0.0) + (i < k - 1 ? fabs(beta[i]) : 0.0);
                lo = dmin_(lo, alpha[i] - rad);
                hi2 = dmax_(hi2, alpha[i] + rad);
            }
            double* y = e == 0 ? ymin : ymax;
            double r;
            if (k <= kLanczosWarm) {
                double ar[kLanczosWarm], br[kLanczosWarm], b2[kLanczosWarm], yr[kLanczosWarm];
#pragma unroll
                for (int i = 0; i < kLanczosWarm; ++i) {
                    ar[i] = i < k ? alpha[i] : 0.0;
                    br[i] = i < k - 1 ? beta[i] : 0.0;
                    b2[i] = br[i] * br[i];
                }
                warp_multisect([&](double x) { return sturm_count8(ar, b2, k, x); }, e == 0 ? 1 : k, lo, hi2);
                r = 0.5 * (lo + hi2);
                tridiag_vec_reg<2>(ar, br, k, r, yr);
                if (wl == 0)
#pragma unroll
                    for (int i = 0; i < kLanczosWarm; ++i)
                        if (i < k) y[i] = yr[i];
            } else {
                warp_multisect([&](double x) { return sturm_count_products(alpha, beta, k, x); }, e == 0 ? 1 : k, lo,
                               hi2);
                r = 0.5 * (lo + hi2);
                if (wl == 0) wk_tridiag_vec(alpha, beta, k, r, y, s3 + 32 * e, s4 + 32 * e);
            }
            if (wl == 0) tot[e] = r;
            if (T > 1) break;
        }
        __syncthreads();
        rmin = tot[0];
        rmax = tot[1];
        for (int d = 0; d < 3; ++d) ritz[d] = 0.0;
        if (on)
            for (int j = 0; j < k; ++j) {
                const double y = ymin[j] + ymax[j];
                const double* vj = V + j * ldv + 3 * b;
#pragma unroll
                for (int d = 0; d < 3; ++d) ritz[d] = fma(y, vj[d], ritz[d]);
            }
    }

    // spectral_bounds (src/hydrodynamics.cpp:224-264). The step's products that
    // do not depend on one another go with the start vector's: D X0 (noise) and
    // D (Fs + Fe) (predictor and, by linearity, upsilon; the product counter
    // keeps the reference's count, which forms D Fs as well).
    // v0: the start vector, replaced by the next step's.
    __device__ __forceinline__ void bounds(double (&v0)[3], int& cache_valid, double& lmin, double& lmax,
                                           const double (&X0)[3], const double (&A)[3], double (&DX0)[3],
                                           double (&DA)[3]) {
        const bool can_warm = cache_valid != 0;
        double v[3] = {v0[0], v0[1], v0[2]}, w[3], ritz[3], rmin, rmax;
        {
            double x3[3][3], y3[3][3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                x3[0][d] = v[d];
                x3[1][d] = X0[d];
                x3[2][d] = A[d];
            }
            apply<3>(x3, y3);
            cnt[C_DX] += 1;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                w[d] = y3[0][d];
                DX0[d] = y3[1][d];
                DA[d] = y3[2][d];
            }
        }
        // (the warm basis is in shared memory, the cold one in global scratch)
        bool cold = !can_warm, have_w = true;
        int k;
        for (;;) {
            k = lanczos(cold ? Vg : area, cold, v, w, have_w);
            if (cold || k >= 4) break;
            start_vector(nullptr, false, v);
            cold = true;
            have_w = false;
        }
        ritz_pair(cold ? Vg : area, k, ritz, rmin, rmax);
        cnt[cold ? C_LZCOLD : C_LZWARM] += 1;
        double s[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) s[d] = on ? fma(0.01, seed[3 * b + d], ritz[d]) : 0.0;
        const double s2 = dot(s, s);
        cache_valid = (s2 > 0.0 && isfinite(s2)) ? 1 : 0;
        if (cache_valid) {
            const double is = rsqrt_refined(s2);
#pragma unroll
            for (int d = 0; d < 3; ++d) v0[d] = s[d] * is;
        } else {
#pragma unroll
            for (int d = 0; d < 3; ++d) v0[d] = on ? seed[3 * b + d] : 0.0;
        }
        lmin = 0.5 * rmin;
        lmax = 1.02 * rmax;
        if (lmin < 1.0e-12) lmin = 1.0e-12;
        if (lmin >= lmax) lmin = lmax * 1.0e-6;
    }

    // ---- Chebyshev square root (src/hydrodynamics.cpp:267-337). Returns the
    // FD error; out = approx D^{1/2} x0. Every cosine of the coefficient sums
    // is cos(pi m / 2P), P = L + 1, with integer m: one table of P + 1 values.
    __device__ __forceinline__ double chebyshev(const double (&x0)[3], const double (&Dx0)[3], double lmin, double lmax,
                                double (&out)[3]) {
        const double x0Dx0 = dot(x0, Dx0);
        double Lr = sqrt(lmax / lmin) * ch.mult + 0.5;
        int L = !(Lr < 2.0e9) ? kMaxCheb : (int)Lr + 1;
        L = L > kMaxCheb ? kMaxCheb : (L < 2 ? 2 : L);
        const double da = 2.0 / (lmax - lmin);
        const double db = -(lmax + lmin) / (lmax - lmin);
        double *ct = area, *sqx = area + kCoefCap, *coef = area + 2 * kCoefCap;
        for (;;) {
            const int P = L + 1;
            for (int m = tid; m <= P; m += TT) ct[m] = cospi((double)m / (2.0 * P));
            __syncthreads();
            for (int k = tid; k < P; k += TT) {
                const int m = 2 * k + 1;
                const double c = m <= P ? ct[m] : -ct[2 * P - m];
                sqx[k] = sqrt(c / da - db / da);
            }
            __syncthreads();
            for (int j = tid; j < P; j += TT) {
                double s = 0.0;
                int m = j;  // j (2k + 1) modulo 4P
                for (int k = 0; k < P; ++k) {
                    const int h = m > 2 * P ? 4 * P - m : m;
                    s = fma(sqx[k], h <= P ? ct[h] : -ct[2 * P - h], s);
                    m += 2 * j;
                    if (m >= 4 * P) m -= 4 * P;
                }
                s *= 2.0 / P;
                coef[j] = j == 0 ? s / 2.0 : s;
            }
            __syncthreads();
            double tp[3], tc[3], o[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                tp[d] = x0[d];
                tc[d] = fma(da, Dx0[d], db * tp[d]);
                o[d] = fma(coef[1], tc[d], coef[0] * tp[d]);
            }
            for (int l = 2; l <= L; ++l) {
                double Dv[3];
                apply1(tc, Dv);
                const double cl = coef[l];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const double tn = fma(2.0, fma(da, Dv[d], db * tc[d]), -tp[d]);
                    tp[d] = tc[d];
                    tc[d] = tn;
                    o[d] = fma(cl, tn, o[d]);
                }
            }
            cnt[C_CHEB] += L;
#pragma unroll
            for (int d = 0; d < 3; ++d) out[d] = o[d];
            const double rr = dot(out, out);  // (its barrier also frees the tables)
            const double fd = fabs(rr - x0Dx0) / x0Dx0;
            if (fd <= ch.fd_tol || L >= kMaxCheb) return fd;
            const int grow = L / 4 > 1 ? L / 4 : 1;
            L = (L + grow) > kMaxCheb ? kMaxCheb : L + grow;
        }
    }
};

// -------------------------------------------------------------- the kernel

template <int T, bool kHi>
__global__ void __launch_bounds__(32 * T, pair_min_blocks(T, kHi)) integrate_pair_kernel(const RunArgs a) {
    extern __shared__ __align__(16) double psm[];
    constexpr int TT = 32 * T;
    const PairLayout lay = pair_layout(a.n_max, T, a.w_pairs);
    DevChain& ch = *reinterpret_cast<DevChain*>(psm + lay.chain);
    PairChain<T> C(a, ch);
    C.red = psm + lay.red;
    C.alpha = psm + lay.alpha;
    C.beta = psm + lay.beta;
    C.ymin = psm + lay.ymin;
    C.ymax = psm + lay.ymax;
    C.tot = psm + lay.tot;
    C.ctl = reinterpret_cast<int32_t*>(psm + lay.ctl);
    C.jcols = reinterpret_cast<uint32_t*>(psm + lay.jcols);
    C.ps = psm + lay.ps;
    C.pq = psm + lay.pq;
    C.xs = psm + lay.xs;
    C.buf = psm + lay.buf;
    C.s3 = psm + lay.s3;
    C.s4 = psm + lay.s4;
    C.area = psm + lay.area;
    C.seed = psm + lay.seed;
    C.Wt = reinterpret_cast<double2*>(psm + lay.w);
    C.ldv = (int)round_up8(a.n_max);
    C.Vg = a.scratch + (int64_t)blockIdx.x * a.scratch_stride;
    C.Lt = C.Vg + (int64_t)kLanczosCold * C.ldv;
    const int tid = threadIdx.x;
    C.tid = tid;
    C.wl = tid & 31;
    C.wi = tid >> 5;
    C.par = 0;
    const uint64_t t_launch = global_ns();

    for (;;) {
        if (tid == 0) {
            const int item = atomicAdd(a.work_counter, 1);
            C.ctl[1] = item >= a.n_work ? -1 : (a.order ? a.order[item] : item);
        }
        __syncthreads();
        const int c = C.ctl[1];
        if (c < 0) break;
        {
            const double* src = reinterpret_cast<const double*>(a.chains + c);
            double* dst = reinterpret_cast<double*>(&ch);
            for (int i = tid; i < (int)(sizeof(DevChain) / 8); i += TT) dst[i] = src[i];
        }
        __syncthreads();
        const int status0 = a.status[c];
        if ((status0 & BDCU_ST_FATAL_MASK) || ch.bad_param) {
            __syncthreads();  // (every thread has read the status word)
            if (tid == 0 && !(status0 & BDCU_ST_FATAL_MASK)) a.status[c] = status0 | BDCU_ST_BAD_PARAM;
            continue;
        }
        const int N = ch.N, n = 3 * N, Ne = (N + 1) & ~1;
        C.N = N;
        C.n = n;
        C.Ne = Ne;
        C.S = pair_lanes(Ne, T);
        // A warp holds G = 16 / S groups of 2S lanes, a group two adjacent beads:
        // lane l is part l / G of group l % G, and its bead the group's first
        // for l < 16, else the second. (Parts in the high lane bits: lanes that
        // share a partner load are then adjacent, and a 16-byte load with up to
        // eight distinct addresses takes two cycles; with the parts in the low
        // bits it takes one per address.)
        C.G = 16 / C.S;
        C.gl = C.wl / C.G;
        const int group = C.wi * C.G + C.wl % C.G;
        C.b = 2 * group + (C.wl >> 4);
        C.seg = C.gl % C.S;
        C.lane_on = group < Ne / 2;
        C.wslot = C.gl * (Ne / 2) + group;
        C.bc = min(C.b, N - 1);
        C.on = C.b < N;
        C.own = C.on && C.seg == 0;
        C.hi = kHi && ch.hstar > 0.0;
        C.status = status0;
        C.np = (Ne / 2 - C.gl + 2 * C.S - 1) / (2 * C.S);
        // (the Cholesky method keeps its factor in the weights' place: three
        // products a step do not repay a table)
        C.nc = ch.hi_method == BDCU_HI_CHOLESKY ? 0 : (int)min((int64_t)C.np, a.w_pairs / (4 * C.S * Ne));
        C.xpar = 0;
        if (C.hi) C.rpy.set(ch.hstar);
        for (int k = 0; k < 8; ++k) C.cnt[k] = 0;
        double* gR = a.R + 3 * ch.bead_off;
        double* gcache = a.cache + 3 * ch.bead_off;
        int cache_valid = (a.cache_mode == BDCU_CACHE_PERSIST) ? a.cache_valid[c] : 0;
        uint32_t ux = (uint32_t)a.rng[3 * c];
        int32_t iy = a.rng[3 * c + 1], sd = a.rng[3 * c + 2];
        double R[3];
        const bool on = C.on, own = C.own;
        const int b = C.b;
        const bool bond_on = b < N - 1;
        for (int d = 0; d < 3; ++d) R[d] = on ? gR[3 * b + d] : 0.0;
        const int nsteps = a.n_steps[c];
        C.noise_start(ux, iy, sd);
        bool drew = false;
        double t = a.t_start[c];
        const double dt = ch.dt;
        const double sqrt2inv = 1.0 / sqrt(2.0);
        const double sqrt_dt = sqrt(dt), inv_n = 1.0 / N;
        double v0[3];  // the Lanczos start vector, kept from step to step
        bool used_cache = false;
        if (kHi && C.hi && ch.hi_method == BDCU_HI_CHEBYSHEV) {
            if (own)
                for (int d = 0; d < 3; ++d) C.seed[3 * b + d] = a.seed_table[3 * b + d] / ch.seed_norm;
            __syncwarp();  // (the lanes of a bead read it back)
            C.start_vector(gcache, cache_valid != 0, v0);
        }
        int step = 0;
        for (; step < nsteps; ++step) {
            if (a.budget_ns > 0) {  // time slice: no new step past the budget
                if (tid == 0) C.ctl[4] = (int64_t)(global_ns() - t_launch) >= a.budget_ns;
                __syncthreads();
                const int stop = C.ctl[4];
                __syncthreads();
                if (stop) break;
            }
            // recenter (src/integrator.cpp:88-93)
            if (ch.update_com) {
                double s[3] = {R[0], R[1], R[2]};
                C.sums(s);
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    if (on) R[d] = R[d] - inv_n * s[d];
            }
            C.stage(C.ps, R);
            double A[3], X0[3], dW[3], DF[3];
            {
                double Fs[3], Fe[3];
                C.forces(C.ps, t, Fs, Fe, true);
#pragma unroll
                for (int d = 0; d < 3; ++d) A[d] = Fs[d] + Fe[d];
            }
            C.noise(ux, iy, X0);
            drew = true;
            // brownian_step (src/mobility.cpp:58-88)
            if (!kHi || !C.hi) {
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    dW[d] = sqrt_dt * X0[d];
                    DF[d] = A[d];
                }
            } else if (ch.hi_method == BDCU_HI_CHOLESKY) {
                double bx[3];
                if (!C.cholesky_noise(X0, bx)) {
                    C.status |= BDCU_ST_NOT_PD;
                    break;
                }
#pragma unroll
                for (int d = 0; d < 3; ++d) dW[d] = sqrt_dt * bx[d];
                C.apply1(A, DF);
                C.cnt[C_DX] += 1;  // (D (Fs + Fe) and, by linearity, the reference's D Fs)
                __syncthreads();
            } else {
                C.build_weights();
                double DX0[3], bx[3], lmin, lmax;
                used_cache = true;
                C.bounds(v0, cache_valid, lmin, lmax, X0, A, DX0, DF);
                const double fd = C.chebyshev(X0, DX0, lmin, lmax, bx);
                if (!(fd <= ch.fd_tol)) {
                    C.status |= BDCU_ST_CHEB_FALLBACK;
                    C.cnt[C_FALLBACK] += 1;
                    C.cnt[C_DX] += 2;  // the reference forms the force products after the factor
                    double *x = C.sb(0), *y = C.sb(1);
                    if (own)
                        for (int d = 0; d < 3; ++d) x[3 * b + d] = X0[d];
                    __syncthreads();
                    bool pd = true;
                    pair_dense(C.Lt, C.ps, N, ch.hstar);
#pragma unroll 1
                    for (int k0 = 0; pd && k0 < n; k0 += kPairPanel) {
                        pd = pair_panel(C.Lt, C.area, n, k0);
                        if (pd) pair_trailing(C.Lt, C.area, n, k0 + kPairPanel);
                    }
                    if (!pd) {
                        C.status |= BDCU_ST_NOT_PD;
                        break;
                    }
                    pair_lower(C.Lt, n, x, y);
#pragma unroll
                    for (int d = 0; d < 3; ++d) bx[d] = on ? y[3 * b + d] : 0.0;
                }
#pragma unroll
                for (int d = 0; d < 3; ++d) dW[d] = sqrt_dt * bx[d];
            }
            // predictor (src/integrator.cpp:96-101)
            double Rp[3], ups[3];
            {
                double K1[9];
                kappa_at(ch, a.arena, t, K1);
#pragma unroll
                for (int r = 0; r < 3; ++r) {
                    const double fl1 = K1[3 * r] * R[0] + K1[3 * r + 1] * R[1] + K1[3 * r + 2] * R[2];
                    Rp[r] = on ? R[r] + dt * (fl1 + 0.25 * DF[r]) + sqrt2inv * dW[r] : 0.0;
                    ups[r] = fl1;
                }
            }
            // upsilon (src/integrator.cpp:107-119): forces at R~; D stays the tensor at R
            C.stage(C.pq, Rp);
            double Fep[3], unused[3];
            C.forces(C.pq, t + dt, unused, Fep, false);
            // solve_connectors (src/integrator.cpp:125-165): the lanes of bead b
            // hold bond b. The first iteration's bonds are those of R~, so that
            // iteration's product D Fb goes with upsilon's D Fe~.
            double bond[3], Fc[3], Fb[3], DFb[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) bond[d] = bond_on ? C.pq[pair_at(b + 1, d)] - C.pq[pair_at(b, d)] : 0.0;
            const double anchor[3] = {C.pq[0], C.pq[2], C.pq[4]};
            // connector forces (src/spring.cpp:183-193) and the bead forces
            auto connector_and_bead_forces = [&]() {
                double* q = C.sb(0);
                const double f = bond_on ? connector_factor(ch, clamped_len(bond[0], bond[1], bond[2])) : 0.0;
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    Fc[d] = f * bond[d];
                    if (own && bond_on) q[3 * b + d] = Fc[d];
                }
                __syncthreads();
                Fb[0] = Fb[1] = Fb[2] = 0.0;
                if (on) C.bead_force(q, Fb);
            };
            connector_and_bead_forces();
            {
                double x2[2][3], y2[2][3];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    x2[0][d] = Fep[d];
                    x2[1][d] = Fb[d];
                }
                C.template apply<2>(x2, y2);
                double K2[9];
                kappa_at(ch, a.arena, t + dt, K2);
#pragma unroll
                for (int r = 0; r < 3; ++r) {
                    DFb[r] = y2[1][r];
                    const double fl2 = K2[3 * r] * Rp[0] + K2[3 * r + 1] * Rp[1] + K2[3 * r + 2] * Rp[2];
                    ups[r] = R[r] + dt * (0.5 * (ups[r] + fl2) + 0.125 * (DF[r] + y2[0][r])) + sqrt2inv * dW[r];
                }
            }
            double dups[3];
            {
                double* q = C.sb(2);
                if (own)
#pragma unroll
                    for (int d = 0; d < 3; ++d) q[3 * b + d] = ups[d];
                __syncthreads();
#pragma unroll
                for (int d = 0; d < 3; ++d) dups[d] = bond_on ? q[3 * (b + 1) + d] - q[3 * b + d] : 0.0;
            }
            double Rprev[3] = {Rp[0], Rp[1], Rp[2]}, Rc[3];
            const int max_iter = 100 * N;
            const double c8 = 0.125 * dt, c4 = 0.25 * dt;
            int lstat = 0;
            for (int iter = 0;; ++iter) {
                if (iter > 0) {  // (the first iteration's Fc, Fb and D Fb are formed above)
                    connector_and_bead_forces();
                    C.apply1(Fb, DFb);
                }
                double* q = C.sb(1);
                if (own)
#pragma unroll
                    for (int d = 0; d < 3; ++d) q[3 * b + d] = DFb[d];
                __syncthreads();
                if (bond_on) {
                    double g[3], qv[3];
                    for (int d = 0; d < 3; ++d)
                        g[d] = dups[d] + c8 * (q[3 * (b + 1) + d] - q[3 * b + d]) + c4 * Fc[d];
                    solve_connector(g, dt, ch, qv, lstat);
                    for (int d = 0; d < 3; ++d) bond[d] = qv[d];
                }
                // R_corr of bead b = anchor + the bonds before it: the group's two
                // bonds together, an inclusive scan over the groups of each
                // warp, the previous group's sum, the totals of the warps before
                double scan[3];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const double o = __shfl_xor_sync(kFull, bond[d], 16);  // the group's other bond
                    double v = bond[d] + o;
                    for (int k = 1; k < C.G; k <<= 1) {
                        const double u = __shfl_up_sync(kFull, v, k);
                        if (C.wl % C.G >= k) v += u;
                    }
                    if (C.wl == C.G - 1) C.tot[3 * C.wi + d] = v;
                    v = __shfl_up_sync(kFull, v, 1);
                    scan[d] = (C.wl % C.G ? v : 0.0) + (C.wl >> 4 ? o : 0.0);
                }
                __syncthreads();
                double e[1] = {0.0};
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    double off = 0.0;
                    for (int w = 0; w < C.wi; ++w) off += C.tot[3 * w + d];
                    Rc[d] = on ? anchor[d] + (off + scan[d]) : 0.0;
                    const double x = Rc[d] - Rprev[d];
                    e[0] += x * x;
                }
                C.sums(e);
                const double incr = sqrt(e[0]) / N;
                C.cnt[C_CORR] += 1;
                if (incr < ch.tol) break;
                if (!(incr == incr) || isinf(incr)) {
                    C.status |= BDCU_ST_NONFINITE;
                    break;
                }
                if (iter >= max_iter) {
                    C.status |= BDCU_ST_NONCONVERGED;
                    C.cnt[C_NONCONV] += 1;
                    break;
                }
#pragma unroll
                for (int d = 0; d < 3; ++d) Rprev[d] = Rc[d];
            }
            C.status |= C.any_bits(lstat);
            if (C.status & BDCU_ST_FATAL_MASK) break;
#pragma unroll
            for (int d = 0; d < 3; ++d) R[d] = Rc[d];
            C.cnt[C_STEPS] += 1;
            t += dt;
        }
        if (used_cache && cache_valid && own)
            for (int d = 0; d < 3; ++d) gcache[3 * b + d] = v0[d];
        if (!(C.status & BDCU_ST_FATAL_MASK) && own)
            for (int d = 0; d < 3; ++d) gR[3 * b + d] = R[d];
        __syncthreads();
        if (tid == 0) {
            if (drew) {  // (lazy seeding belongs to the first draw)
                a.rng[3 * c] = (int32_t)ux;
                a.rng[3 * c + 1] = iy;
                a.rng[3 * c + 2] = sd;
            }
            a.cache_valid[c] = cache_valid;
            a.status[c] = C.status;
            int64_t* cc = reinterpret_cast<int64_t*>(a.counters + c);
            for (int k = 0; k < 8; ++k) cc[k] += (int64_t)C.cnt[k];
            if (a.steps_done) a.steps_done[c] = step;
            if (a.t_end) a.t_end[c] = t;
        }
        __syncthreads();
    }
}

}  // namespace bdcu
