"""The plain form's results follow from the chain alone: not from the launch
shape, the other chains of the launch or the entry point, bit for bit."""
import numpy as np
import pytest

import bdsim_b200 as B
from bdsim_b200 import _abi, workloads
from bdsim_b200.params import DelSMethod

pytestmark = pytest.mark.gpu


def gauss(N, copies, method=DelSMethod.Chebyshev, form="plain"):
    p, s = workloads.batched_cheb_phys(N)
    p.hi_method = method
    R0 = [B.gaussian_chain(N, bond_std=1.0, seed=i) for i in range(copies)]
    return B.Ensemble([p] * copies, [s] * copies, R0, [(1, -1, 5 + i) for i in range(copies)], form=form)


@pytest.mark.parametrize("N,copies,method", [(10, 2048, DelSMethod.Chebyshev), (20, 2048, DelSMethod.Chebyshev),
                                             (100, 300, DelSMethod.Chebyshev), (256, 148, DelSMethod.Chebyshev),
                                             (10, 64, DelSMethod.Cholesky), (70, 64, DelSMethod.Cholesky)])
def test_autotune_changes_no_result(N, copies, method):
    ends = []
    for tune in (False, True):
        ens = gauss(N, copies, method)
        if tune:
            assert all(b["tuned"] == 1 for b in ens.autotune(probe_steps=2))
        ens.advance(0.0, 2, _abi.CACHE_RESET_PER_CALL)
        ends.append(ens.R.cpu().numpy())
    assert np.array_equal(ends[0], ends[1])


@pytest.mark.parametrize("form", ["plain", "mixed"])
@pytest.mark.parametrize("N,other", [(66, 128), (101, 127), (110, 128), (150, 250), (258, 500)])
def test_cholesky_does_not_depend_on_the_other_chains(form, N, other):
    """The blocked factorisation (3N >= 300) among longer chains of its bucket."""
    ends = []
    for Ns in ([N], [other, N, other]):
        phys, sims, R0 = [], [], []
        for n in Ns:
            p, s = workloads.batched_cheb_phys(n)
            p.hi_method = DelSMethod.Cholesky
            phys.append(p)
            sims.append(s)
            R0.append(B.gaussian_chain(n, bond_std=1.0, seed=n))
        ens = B.Ensemble(phys, sims, R0, [(1, -1, n) for n in Ns], form=form)
        ens.advance(0.0, 2, _abi.CACHE_RESET_PER_CALL)
        ends.append(ens.positions()[Ns.index(N)])
    assert np.array_equal(ends[0], ends[1])


def both_methods(specs):
    """One plain ensemble of (N, method, copies) groups."""
    phys, sims, R0 = [], [], []
    for N, method, copies in specs:
        p, s = workloads.batched_cheb_phys(N)
        p.hi_method = method
        phys += [p] * copies
        sims += [s] * copies
        R0 += [B.gaussian_chain(N, bond_std=1.0, seed=100 * N + i) for i in range(copies)]
    return B.Ensemble(phys, sims, R0, [(1, -1, 5 + i) for i in range(len(R0))], form="plain")


def test_a_cholesky_chain_leaves_the_chebyshev_launch_as_it_was():
    """A Cholesky chain of N <= 64 keeps its factor in shared memory, which its
    Chebyshev neighbours do not pay for."""
    cheb, chol = DelSMethod.Chebyshev, DelSMethod.Cholesky
    alone = both_methods([(50, cheb, 500)])
    mixed = both_methods([(50, cheb, 500), (64, chol, 1)])
    want = alone.plan()[0]
    got = [b for b in mixed.plan() if b["n_chains"] == 500]
    assert len(got) == 1
    for k in ("block", "grid", "smem_bytes", "max_beads"):
        assert got[0][k] == want[k], k
    one = both_methods([(64, chol, 1)])
    one.rng.copy_(mixed.rng[500:])
    for ens in (alone, mixed, one):
        ens.advance(0.0, 2, _abi.CACHE_RESET_PER_CALL)
    end = mixed.positions()
    assert all(np.array_equal(a, b) for a, b in zip(end, alone.positions()))
    assert np.array_equal(end[500], one.positions()[0])


def test_a_plan_names_each_bucket_once():
    """The plain form launches both methods apart in every size class."""
    cheb, chol = DelSMethod.Chebyshev, DelSMethod.Cholesky
    groups = [(N, m, k) for k, N in enumerate((20, 100, 200, 300, 400), 1) for m in (cheb, chol)] + [(520, cheb, 1)]
    plan = both_methods(groups).plan()
    by_id = {b["bucket"]: b for b in plan}
    assert len(by_id) == len(plan) == 8
    assert sum(b["n_chains"] for b in plan) == sum(g[2] for g in groups)
    # the chains without the Cholesky method keep the ids of a plan without it
    for b in both_methods([g for g in groups if g[1] == cheb and g[0] <= 512]).plan():
        for k in ("n_chains", "min_beads", "max_beads", "block"):
            assert by_id[b["bucket"]][k] == b[k], (b["bucket"], k)
    assert sorted(b["bucket"] for b in both_methods([g for g in groups if g[1] == chol]).plan()) == [4, 5, 6, 7]


def run_static(phys, sims, R0, rng, steps, form, pad=0):
    """bdcu_run_static from t = 0; pad: unused doubles at the arena's end. Returns
    its code and the final positions."""
    import torch
    n, dev = len(R0), torch.device("cuda", 0)
    prec, srec, arena = _abi.pack_batch(phys, sims, [len(r) for r in R0])
    arena = np.concatenate([arena, np.zeros(pad)])
    R = torch.from_numpy(np.concatenate(R0)).to(dev)
    state = torch.tensor(rng, dtype=torch.int32, device=dev)
    cache, t0 = torch.zeros_like(R), torch.zeros(n, dtype=torch.float64, device=dev)
    valid, status = (torch.zeros(n, dtype=torch.int32, device=dev) for _ in range(2))
    k = torch.full((n,), steps, dtype=torch.int32, device=dev)
    cnt = torch.zeros((n, 8), dtype=torch.int64, device=dev)
    ctx = B.Context(0)
    ctx.use_stream()
    rc = ctx.lib.bdcu_run_static(ctx.h, n, prec, srec, arena.ctypes.data_as(_abi.c_double_p), arena.size,
                                 _abi.dptr(R), _abi.dptr(state), _abi.dptr(cache), _abi.dptr(valid), _abi.dptr(t0),
                                 _abi.dptr(k), _abi.dptr(status), _abi.dptr(cnt),
                                 _abi.FORM_PLAIN_FP64 if form == "plain" else _abi.FORM_MIXED_FP32,
                                 _abi.CACHE_RESET_PER_CALL)
    torch.cuda.synchronize()
    return rc, R.cpu().numpy()


@pytest.mark.parametrize("form", ["plain", "mixed"])
def test_static_entry_point_runs_the_same_kernels(form):
    phys, sims, R0 = [], [], []
    for N, method, hstar in [(10, "Chebyshev", 0.25), (50, "Chebyshev", 0.25), (64, "Cholesky", 0.25),
                             (30, "Cholesky", 0.25), (100, "Chebyshev", 0.25), (100, "Cholesky", 0.25),
                             (250, "Chebyshev", 0.25), (40, "Chebyshev", 0.0)]:
        p, s = workloads.batched_cheb_phys(N)
        p.hi_method, p.hstar = DelSMethod[method], hstar
        phys.append(p)
        sims.append(s)
        R0.append(B.gaussian_chain(N, bond_std=1.0, seed=N))
    rng = [(1, -1, 5 + i) for i in range(len(R0))]
    ens = B.Ensemble(phys, sims, R0, rng, form=form)
    ens.advance(0.0, 2, _abi.CACHE_RESET_PER_CALL)
    rc, got = run_static(phys, sims, R0, rng, 2, form)
    assert rc == 0 and np.array_equal(got, ens.R.cpu().numpy())


def falling_back(N, copies, fd_err_max=-1.0, method=DelSMethod.Chebyshev):
    """Chains whose series starts at its largest order and, for a negative bound
    on its error, falls back to the Cholesky factor in every step."""
    p, s = workloads.batched_cheb_phys(N)
    p.ncheb_multiplier, p.fd_err_max, p.hi_method = 1e4, fd_err_max, method
    R0 = [B.gaussian_chain(N, bond_std=1.0, seed=N)] * copies
    return B.Ensemble([p] * copies, [s] * copies, R0, [(1, -1, 7)] * copies, form="plain")


@pytest.mark.parametrize("N", [64, 65, 99, 100, 101, 128, 170, 257])
def test_fallback_sizes(port, N):
    """The blocked factorisation (3N >= 300) against the oracle, and the same bits
    among enough chains that the launch caches fewer weights (the factor is staged
    in their place)."""
    p, s = workloads.batched_cheb_phys(N)
    p.ncheb_multiplier, p.fd_err_max = 1e4, -1.0
    s.time_start, s.time_end = 0.0, s.dt
    R0 = B.gaussian_chain(N, bond_std=1.0, seed=N)
    want, _, _, cnt = port.integrate(R0, p, s, (1, -1, 7))
    ends = []
    for copies in (1, 450):
        ens = falling_back(N, copies)
        ens.advance(0.0, 2, _abi.CACHE_RESET_PER_CALL)
        assert cnt["cheb_fallbacks"] == 2 and int(ens.counters[0, 6]) == 2
        ends.append(ens.positions()[0])
    assert np.max(np.abs(ends[0] - want)) <= 1e-10 * max(1.0, np.max(np.abs(want)))
    assert np.array_equal(ends[0], ends[1])


def test_fallback_costs_no_more_than_the_cholesky_method():
    """Both factor one tensor; column by column the fallback's factor took 17 times
    the Cholesky method's whole step."""
    import torch

    def ms(ens):
        best, R = 1e9, ens.R.clone()
        for _ in range(4):
            ens.R.copy_(R)
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            ens.advance(0.0, 1, _abi.CACHE_RESET_PER_CALL)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    factor = ms(falling_back(300, 148)) - ms(falling_back(300, 148, fd_err_max=1.0))
    assert factor <= 4.0 * ms(falling_back(300, 148, method=DelSMethod.Cholesky))


@pytest.mark.parametrize("hstar", [0.25, 0.0])
@pytest.mark.parametrize("N,blocks", [(2, 12), (3, 6), (4, 6), (5, 8), (64, 6)])
def test_many_short_chains_fill_the_sms(hstar, N, blocks):
    """Short chains, and chains without HI, in numbers: more blocks on an SM than a
    few of them get (three of four warps), and the same bits as alone, whatever the
    launch's width and build."""
    ends = []
    for copies in (3, 2000):
        p, s = workloads.batched_cheb_phys(N)
        p.hstar = hstar
        R0 = [B.gaussian_chain(N, bond_std=1.0, seed=i % 3) for i in range(copies)]
        ens = B.Ensemble([p] * copies, [s] * copies, R0, [(1, -1, 5 + i % 3) for i in range(copies)], form="plain")
        grid = ens.plan()[0]["grid"]
        assert grid == copies if copies < 2000 else grid >= min(2000, 148 * (3 if N > 4 and hstar > 0.0 else blocks))
        ens.advance(0.0, 4, _abi.CACHE_RESET_PER_CALL)
        ends.append(ens.positions())
    assert all(np.array_equal(r, ends[0][i % 3]) for i, r in enumerate(ends[1]))


def test_mixed_fallback_costs_no_more_than_twice_the_cholesky_method():
    """N = 50: a factor of the team kernel (2.9 ms while each column waited for L2)
    against a step of the Cholesky method on the block kernel."""
    import torch

    def ms(method, fd_err_max):
        p, s = workloads.batched_cheb_phys(50)
        p.ncheb_multiplier, p.fd_err_max, p.hi_method = 1e4, fd_err_max, method
        ens = B.Ensemble([p], [s], [B.gaussian_chain(50, bond_std=1.0, seed=1)], [(1, -1, 7)], form="mixed")
        best, R = 1e9, ens.R.clone()
        for _ in range(6):
            ens.R.copy_(R)
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            ens.advance(0.0, 1, _abi.CACHE_RESET_PER_CALL)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    factor = ms(DelSMethod.Chebyshev, -1.0) - ms(DelSMethod.Chebyshev, 1.0)
    assert factor <= 2.0 * ms(DelSMethod.Cholesky, 1.0)


@pytest.mark.parametrize("N,method", [(400, DelSMethod.Cholesky), (430, DelSMethod.Chebyshev)])
def test_static_entry_point_asks_for_what_its_kernels_take(N, method):
    """One block's factor (11.6 MB, 13.3 MB) fits the 16 MiB array; a dense tensor
    beside it, which no kernel forms, did not."""
    p, s = workloads.batched_cheb_phys(N)
    p.hi_method = method
    R0 = [B.gaussian_chain(N, bond_std=1.0, seed=1)]
    ens = B.Ensemble([p], [s], R0, [(1, -1, 5)], form="plain")
    ens.advance(0.0, 1, _abi.CACHE_RESET_PER_CALL)
    rc, got = run_static([p], [s], R0, [(1, -1, 5)], 1, "plain")
    assert rc == 0 and np.array_equal(got, ens.R.cpu().numpy())


def test_static_entry_point_at_its_limit():
    """A plain batch whose parameters leave room for the general kernel's scratch but
    not for the pair kernel's still runs, to rounding."""
    p, s = workloads.batched_cheb_phys(100)
    R0 = [B.gaussian_chain(100, bond_std=1.0, seed=1)]
    ens = B.Ensemble([p], [s], R0, [(1, -1, 5)], form="plain")
    ens.advance(0.0, 1, _abi.CACHE_RESET_PER_CALL)
    want = ens.R.cpu().numpy()
    ran = {}
    for kb in (0, 15600, 15630, 15700, 16300):
        rc, got = run_static([p], [s], R0, [(1, -1, 5)], 1, "plain", pad=128 * kb)
        ran[kb] = (rc, np.array_equal(got, want))
        if rc == 0:
            assert np.max(np.abs(got - want)) <= 1e-10 * max(1.0, np.max(np.abs(want)))
        else:
            assert rc == 5  # BDCU_E_LIMIT
    assert ran[0] == (0, True) and ran[16300][0] == 5
    assert any(rc == 0 and not same for rc, same in ran.values())
