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
