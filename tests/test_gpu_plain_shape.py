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
