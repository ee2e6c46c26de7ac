"""Chains whose beads lie close together under strong HI: the tensor's spectrum spreads
over many decades and a Lanczos basis loses its orthogonality within a few steps. Steps
from a cold start, with the spectral bounds of a 30-step run, against the oracle."""
import numpy as np
import pytest

import bdsim_b200 as B
from bdsim_b200 import _abi, workloads
from bdsim_b200.params import Rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,tol,steps", [("plain", 1e-10, 1), ("plain", 1e-10, 3), ("mixed", 1e-4, 1)])
@pytest.mark.parametrize("N", [24, 30, 35, 50, 100, 200])
@pytest.mark.parametrize("hstar,scale", [(0.25, 0.1), (0.25, 0.2), (0.5, 0.05), (0.5, 0.15)])
def test_cold_bounds(port, N, hstar, scale, form, tol, steps):
    """Tolerances per call as in the parity tests. The counters show the bounds: wrong
    ones change the order of the Chebyshev series."""
    p, s = workloads.batched_cheb_phys(N)
    p.hstar = hstar
    s.time_start, s.time_end = 0.0, (steps - 1) * s.dt
    R0 = scale * B.gaussian_chain(N, bond_std=1.0, seed=N)
    g = Rng(7)
    out, status, cnt = B.integrate_many([R0], p, s, [g], form=form)
    want, _, want_status, want_cnt = port.integrate(R0, p, s, (1, -1, 7))
    assert int(status[0]) == int(want_status)
    assert np.max(np.abs(out[0] - want)) <= tol * max(1.0, float(np.max(np.abs(want))))
    assert abs(cnt[0]["cheb_terms"] - want_cnt["cheb_terms"]) <= steps
