// pair_layout.h -- sizes of the pair kernel's shared and global scratch
// (integrator_pair.cuh), shared by the host launch code and the kernel.
//
// The pair kernel is the FP64 plain form for chains of up to 512 beads (64 with
// the Cholesky method): one chain per thread block of T warps, S lanes per bead.
#pragma once

#include "integrator.cuh"

namespace bdcu {

constexpr int kPairMaxN = 512;
// Cholesky-method chains up to this size factor D in shared memory (150 KB at 64
// beads); larger ones run on the block kernel.
constexpr int kPairCholMaxN = 64;
__host__ __device__ inline int64_t pair_factor_doubles(int N) { return 9 * (int64_t)N * (N + 1) / 2; }

// Blocks per SM a shape's registers and shared memory are sized for. 12 to 16
// warps per SM: 168 registers per thread up to T = 4, 128 at T = 8 and 16. hi:
// whether the launch has a chain with HI; the build without leaves its code out and
// runs 8 blocks of T = 4 (64 registers) instead of 3.
__host__ __device__ constexpr int pair_min_blocks(int T, bool hi) {
    return T <= 4 ? (hi || T < 4 ? 12 / T : 8) : T == 8 ? 2 : 1;
}

// Warps per chain of buckets 0..3 (N <= 64, 128, 256, 512; fewer in launches of the
// shortest chains), and of the Cholesky method's. One shape must serve any number of
// chains (6 steps; 100 and 3000 chains): N = 130 on 8 warps 4.51 and 49.2 ms, on 16 3.31
// and 43.9; N = 256 13.2 and 123, 9.2 and 121; N = 128 on 8 2.88 and 29.1, on 16 2.58 and
// 33.2, on 4 4.07 and 32.7; N = 64 on 4 0.81 and 7.5, on 8 0.94 and 8.5.
constexpr int kPairWarps[4] = {4, 8, 16, 16};
constexpr int kPairCholWarps = 4;

struct PairLayout {
    int64_t chain, red, alpha, beta, ymin, ymax, tot, ctl, jcols, ps, pq, xs, buf, s3, s4, seed, area, w, total;  // in doubles
};

// Lanes per bead of a chain of Ne beads (rounded up to even) on T warps: the
// largest power of two (at most 16) that leaves every bead its lanes.
__host__ __device__ inline int pair_lanes(int Ne, int T) {
    int S = 1;
    while (S < 16 && 2 * S * Ne <= 32 * T) S *= 2;
    return S;
}

// Cached weights a chain of N beads takes when all are kept: two beads per
// group of 2S lanes against the lane's share of the partner pairs, rounded up
// to the same number for every lane.
__host__ __device__ inline int64_t pair_weights(int N, int T) {
    const int Ne = (N + 1) / 2 * 2, S = pair_lanes(Ne, T);
    return (int64_t)((Ne / 2 + 2 * S - 1) / (2 * S)) * 4 * S * Ne;
}

// Layout for chains of up to n_max/3 beads and w_pairs cached pair weights
// (two doubles each).
__host__ __device__ inline PairLayout pair_layout(int n_max, int T, int64_t w_pairs) {
    PairLayout s;
    const int64_t N = n_max / 3, Ne = (N + 1) / 2 * 2, n8 = round_up8(n_max);
    int64_t o = 0;
    s.chain = o; o += round_up8((int64_t)(sizeof(DevChain) + 7) / 8);
    s.red = o;   o += 2 * 32 * (int64_t)T;  // two buffers of 32 values x T warps
    s.alpha = o; o += 32;
    s.beta = o;  o += 32;
    s.ymin = o;  o += 32;
    s.ymax = o;  o += 32;
    s.tot = o;   o += 3 * (int64_t)T + (T & 1);
    s.ctl = o;   o += 4;
    s.jcols = o; o += 16;
    s.ps = o;    o += 3 * Ne;
    s.pq = o;    o += 3 * Ne;
    s.xs = o;    o += 9 * Ne;
    s.buf = o;   o += 9 * Ne;  // neighbour-exchange buffers (3 x 3N)
    s.s3 = o;    o += Ne > 64 ? Ne : 64;
    s.s4 = o;    o += Ne > 64 ? Ne : 64;
    s.seed = o;  o += 3 * Ne;  // normalised default Lanczos seed
    // warm Lanczos basis; the Chebyshev cosine, node and coefficient tables
    // (3 x kCoefCap) share it, as the basis is dead once the bounds are known
    const int64_t v = (int64_t)kLanczosWarm * n8;
    s.area = o;  o += v > 3 * kCoefCap ? v : 3 * (int64_t)kCoefCap;
    s.w = o;     o += 2 * w_pairs;
    s.total = o;
    return s;
}

// Pair weights a block of shape T caches: all of the largest chain's when they
// fit the block's share of an SM's shared memory, else as many as fit (the rest
// is evaluated again in every product). The share is what the launch's `blocks`
// leave an SM. The split changes no result.
__host__ inline int64_t pair_cached(int n_max, int T, int blocks, int sm_count, size_t max_smem) {
    int per_sm = (blocks + sm_count - 1) / sm_count;
    if (per_sm > pair_min_blocks(T, true)) per_sm = pair_min_blocks(T, true);
    const int64_t share = ((int64_t)max_smem + 1024) / per_sm - 1024;
    const int64_t room = (share / 8 - pair_layout(n_max, T, 0).total) / 2;
    const int64_t all = pair_weights(n_max / 3, T);
    return room <= 0 ? 0 : room < all ? room : all;
}

// Per-block global scratch (doubles): cold Lanczos basis, fallback factor.
__host__ __device__ inline int64_t pair_scratch_doubles(int n_max) {
    return (int64_t)kLanczosCold * round_up8(n_max) + (int64_t)n_max * n_max;
}

}  // namespace bdcu
