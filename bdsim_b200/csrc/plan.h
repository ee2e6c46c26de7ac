// plan.h -- which kernel and launch shape a chain gets: shared by bdcu_run's
// launch plans (api.cu) and the static-scratch entry point (static_scratch.cu),
// so that both run every chain on the same kernel.
#pragma once

#include <algorithm>

#include "ctx.h"
#include "pair_layout.h"
#include "team_layout.h"

namespace bdcu {

// Bucket of a chain for `form` (bucket ids as in ctx.h). pair: whether the
// plain form's pair kernel may be used (the static-scratch entry point goes
// without where its array does not hold the pair kernel's scratch).
inline int bucket_of(const DevChain& c, int form, bool pair = true) {
    const bool chol = c.hstar > 0.0 && c.hi_method == BDCU_HI_CHOLESKY;
    const bool mixed = form == BDCU_FORM_MIXED_FP32;
    static_assert(kPairMaxN == kTeamMaxN, "team and pair buckets share their bead ranges");
    if (!mixed && pair && chol && c.N <= kPairCholMaxN) return kPairCholBucket;
    if (!chol && c.N <= kTeamMaxN && (mixed || pair)) {
        const int T = team_warps_for(c.N);
        return T == 1 ? 0 : T == 2 ? 1 : T == 4 ? 2 : 3;
    }
    for (int b = kFirstBlockBucket; b < 7; ++b)
        if (c.N <= kBucketBeads[b]) return b;
    return 7;
}

// The kernel of a bucket (BDCU_KERNEL_*, kKernelPair).
inline int bucket_kernel(int id, int form) {
    if (id == kPairCholBucket) return kKernelPair;
    if (id >= kFirstBlockBucket) return BDCU_KERNEL_BLOCK;
    return form == BDCU_FORM_MIXED_FP32 ? (int)BDCU_KERNEL_TEAM : kKernelPair;
}

// The pair kernel's warps per chain in a launch over `chains` chains of up to
// n_max/3 beads. Its sums run in the order of the lanes per bead and the warps, so
// that a chain's result does not depend on the launch it is in the warps follow
// from its bucket (not from a timing). Chains that have their 16 lanes per bead on
// fewer warps (N = 2 on one, N <= 4 on two) end in the same bits there: the further
// warps would add zeros. They take the fewer warps where the chains outnumber the
// blocks of four warps on the SMs (3 each); below that one chain's latency counts.
// (16384 dumbbells, 10 steps: with HI 12.5 -> 5.3 ms, without 2.97 -> 0.94.)
inline int pair_warps(int id, int n_max, int chains, int sm_count) {
    if (id == kPairCholBucket) return kPairCholWarps;
    if (chains > 3 * sm_count && n_max <= 12) return n_max <= 6 ? 1 : 2;
    return kPairWarps[id];
}

// Whether such a launch on T warps takes the build with HI: a launch without it
// takes the other one at T = 4 where it has more chains than the build with HI has
// blocks on the SMs (both give a chain the same bits). (4096 free-draining chains,
// 10 steps: N = 5 0.86 -> 0.56 ms, N = 64 2.09 -> 1.83; 400 chains of N = 64 were
// 0.27 -> 0.31.)
inline bool pair_hi(int T, bool hi, int chains, int sm_count) { return hi || T != 4 || chains <= 3 * sm_count; }

// Pair weights in shared memory (16 bytes each) of a block of a pair bucket's
// launch over `chains` chains; a Cholesky bucket's factor takes their place.
inline int64_t pair_shared(int id, int T, int n_max, bool need_lz, int chains, int sm_count, size_t max_smem) {
    if (id == kPairCholBucket) return (pair_factor_doubles(n_max / 3) + 1) / 2;
    return need_lz ? pair_cached(n_max, T, chains, sm_count, max_smem) : 0;
}

#define BDCU_TEAM_SHAPE_SWITCH(T, Q, EXPR, FALLBACK)            \
    (T == 1 && Q == 2)   ? EXPR(1, 2)                            \
    : (T == 2 && Q == 1) ? EXPR(2, 1)                            \
    : (T == 2 && Q == 2) ? EXPR(2, 2)                            \
    : (T == 4 && Q == 1) ? EXPR(4, 1)                            \
    : (T == 4 && Q == 2) ? EXPR(4, 2)                            \
    : (T == 8 && Q == 1) ? EXPR(8, 1)                            \
    : (T == 8 && Q == 2) ? EXPR(8, 2)                            \
                         : FALLBACK

// Shared memory of a team-kernel block of shape (T, Q) for chains of up to
// n_max/3 beads with w_pairs cached weights per team (-1: no such shape).
inline int64_t team_smem(int T, int Q, int n_max, int64_t w_pairs) {
#define BDCU_SMEM(t, q) (team_smem_bytes<t, q>(n_max, w_pairs))
    return BDCU_TEAM_SHAPE_SWITCH(T, Q, BDCU_SMEM, (int64_t)-1);
#undef BDCU_SMEM
}

inline int teams_per_cta(int T, int Q) {
#define BDCU_TPC(t, q) TeamCfg<t, q>::kTeamsPerCta
    return BDCU_TEAM_SHAPE_SWITCH(T, Q, BDCU_TPC, 1);
#undef BDCU_TPC
}

// Cached weights per team of shape (T, Q) in a launch over `chains` chains.
inline int64_t team_weights(int T, int Q, int n_max, int chains, int sm_count, size_t max_smem) {
    const int blocks = (chains + teams_per_cta(T, Q) - 1) / teams_per_cta(T, Q);
#define BDCU_WTS(t, q) (team_cached<t, q>(n_max, blocks, sm_count, max_smem))
    return BDCU_TEAM_SHAPE_SWITCH(T, Q, BDCU_WTS, (int64_t)0);
#undef BDCU_WTS
}

// Whether (T, Q) is a compiled team shape that holds chains of `beads`.
inline bool team_shape_fits(int T, int Q, int beads) {
    for (int i = 0; i < kNumTeamShapes; ++i)
        if (kTeamShapes[i][0] == T && kTeamShapes[i][1] == Q) return beads <= 32 * T * Q;
    return false;
}

// Threads per block of the block kernel's heuristic shape: one thread per row
// of D up to 512.
inline int widest_block(int n_max) {
    int b = ((std::min(n_max, 512) + 31) / 32) * 32;
    return b < 64 ? 64 : b;
}

}  // namespace bdcu
