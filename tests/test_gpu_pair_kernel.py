"""The pair kernel (plain form, one chain per block with FP64 pair weights) and
the cached pair weights of the mixed form, at the sizes where lanes, segments,
padding and the cached range change, against the oracle.

Tolerances as in test_gpu_parity: 1e-10 per plain call of a few steps, 1e-4 per
mixed call; RNG streams and counters exactly. Forces: 1e-12 relative to the
largest force (FP64 sums of up to N terms in another order)."""
import numpy as np
import pytest

import bdsim_b200 as B
from bdsim_b200 import _abi, workloads
from bdsim_b200.params import DelSMethod, EV, Rng, SimParams

pytestmark = pytest.mark.gpu

CALL_TOL = 1e-10
MIXED_TOL = 1e-4
FORCE_TOL = 1e-12


def rel(a, b):
    return float(np.max(np.abs(np.asarray(a) - np.asarray(b))) / max(1.0, float(np.max(np.abs(b)))))


def span(sim, steps):
    s = SimParams()
    s.dt, s.implicit_loop_tol = sim.dt, sim.implicit_loop_tol
    s.time_start, s.time_end = 0.0, (steps - 1) * sim.dt
    return s


def chain(kind, N, seed):
    if kind == "gauss":
        p, s = workloads.batched_cheb_phys(N)
        return p, s, B.gaussian_chain(N, bond_std=1.0, seed=seed)
    if kind == "lj":
        phys, sims, R0, _ = workloads.uneven_wlc(1, seed=seed, Ns=[N])
        return phys[0], sims[0], R0[0]
    p, s = workloads.stiff_large_phys(N)  # SDK with a phi table, bending
    return p, s, B.initial.fene_fraenkel_bending_chain(N, 1.0, 0.1, 5.0, seed=seed)


def against_oracle(port, p, s, R0, seed, steps, form):
    g = Rng(seed)
    out, status, cnt = B.integrate_many([R0], p, span(s, steps), [g], form=form)
    want, st, pst, pcnt = port.integrate(R0, p, span(s, steps), (1, -1, seed))
    assert g.state() == st
    assert int(status[0]) == int(pst)
    assert rel(out[0], want) <= (CALL_TOL if form == "plain" else MIXED_TOL)
    if form == "plain":
        for k in ("steps", "corrector_iters", "lanczos_cold", "lanczos_warm", "cheb_fallbacks", "nonconverged"):
            assert cnt[0][k] == pcnt[k], k


# lanes per bead 16 .. 1 on each warp count, odd sizes, both sides of each bucket
SIZES = [2, 3, 5, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257]


@pytest.mark.parametrize("N", SIZES + [511, 512, 513])
@pytest.mark.parametrize("kind", ["gauss", "lj"])
def test_plain_chebyshev_sizes(port, N, kind):
    p, s, R0 = chain(kind, N, 11 + N)
    against_oracle(port, p, s, R0, 5 + N, 3 if N <= 128 else 2, "plain")


@pytest.mark.parametrize("N", [2, 3, 4, 10, 16, 17, 33, 63, 64, 65])
def test_plain_cholesky_sizes(port, N):
    """In shared memory up to N = 64, on the block kernel above."""
    p, s, _ = chain("gauss", N, 0)
    p.hi_method = DelSMethod.Cholesky
    against_oracle(port, p, s, B.gaussian_chain(N, bond_std=1.0, seed=N), 5 + N, 3, "plain")


@pytest.mark.parametrize("N", [2, 3, 5, 61, 62, 63, 64, 65, 109, 126, 127, 128, 130, 253])
def test_mixed_sizes(port, N):
    """Every remainder modulo the four partners of a cached step, and sizes
    whose weights are cached in part."""
    p, s, R0 = chain("gauss", N, 11 + N)
    against_oracle(port, p, s, R0, 5 + N, 3, "mixed")


@pytest.mark.parametrize("form,N,copies", [("plain", 50, 600), ("plain", 97, 300), ("plain", 150, 300),
                                           ("mixed", 120, 400), ("mixed", 200, 300)])
def test_cached_share_changes_no_result(form, N, copies):
    """A chain alone (all the shared memory for its weights) and among enough
    chains to fill the SMs ends in the same bits."""
    p, s, R0 = chain("gauss", N, 3)
    ends = []
    for n in (1, copies):
        ens = B.Ensemble([p] * n, [s] * n, [R0] * n, [(1, -1, 9)] * n, form=form)
        ens.advance(0.0, 3, _abi.CACHE_RESET_PER_CALL)
        ends.append(ens.positions())
    assert np.array_equal(ends[0][0], ends[1][0])
    assert all(np.array_equal(ends[1][0], r) for r in ends[1])


@pytest.mark.parametrize("kind,N", [("gauss", 2), ("gauss", 50), ("gauss", 129), ("lj", 33), ("lj", 128), ("sdk", 40),
                                    ("sdk", 257)])
def test_forces_sizes(port, kind, N):
    p, _, R0 = chain(kind, N, 7)
    got, want = B.total_force(R0, p), port.total_force(R0, p)
    assert np.max(np.abs(got - want)) <= FORCE_TOL * max(1.0, float(np.max(np.abs(want))))


@pytest.mark.parametrize("form", ["plain", "mixed"])
def test_no_steps_leave_the_stream_unseeded(form):
    p, s, R0 = chain("gauss", 20, 1)
    ens = B.Ensemble([p] * 2, [s] * 2, [R0] * 2, [(1, -1, 4), (1, -1, -4)], form=form)
    ens.advance(0.0, [0, 1], _abi.CACHE_RESET_PER_CALL)
    assert ens.rng_states()[0] == (1, -1, 4) and ens.rng_states()[1] != (1, -1, -4)
    assert np.array_equal(ens.positions()[0], R0)


def test_warm_vector_of_any_length(port):
    """A caller's warm-start vector is normalised first."""
    import torch
    p, s, R0 = chain("gauss", 40, 2)
    cache = [np.zeros(120), 0]
    R1, st, _, _ = port.integrate(R0, p, span(s, 1), (1, -1, 3), cache=cache)
    want, _, _, _ = port.integrate(R1, p, span(s, 1), st, cache=[3.0 * cache[0], 1])
    ens = B.Ensemble([p], [s], [R1], [st], form="plain")
    ens.cache.copy_(torch.from_numpy(3.0 * cache[0]))
    ens.cache_valid.fill_(1)
    ens.advance(0.0, 1, _abi.CACHE_PERSIST)
    assert rel(ens.positions()[0], want) <= CALL_TOL


@pytest.mark.parametrize("method", [DelSMethod.Chebyshev, DelSMethod.Cholesky])
def test_coincident_beads_at_small_hstar(port, method):
    """Two beads in one place: their separation is clamped to 1e-6, which at
    h* = 1e-8 is a far pair."""
    p, s, R0 = chain("gauss", 9, 4)
    R0[6] = R0[2]
    p.hstar, p.hi_method = 1e-8, method
    against_oracle(port, p, s, R0, 8, 1, "plain")
