"""SDK excluded volume where its two ranges overlap: with min_cutoff above
2^(1/6) dstar (dstar below 0.62 at the default 0.7) a pair between the two
feels the constant core and the attraction together
(ExcludedVolume::sdk_factor, src/excluded_volume.cpp:48-58).

Tolerances as in test_gpu_pair_kernel: forces 1e-12 relative to the largest
force, 1e-10 per plain call, 1e-4 per mixed call."""
import numpy as np
import pytest

import bdsim_b200 as B
from bdsim_b200 import flows
from bdsim_b200.params import DelSMethod, EV, PhysParams, Rng, SimParams, Spring

pytestmark = pytest.mark.gpu

# below 2^(1/6) 0.5 = 0.5612, between it and min_cutoff = 0.7, above both
SEPARATIONS = [0.55, 0.5612, 0.5613, 0.60, 0.65, 0.69, 0.72]


def sdk_chain(N, method=DelSMethod.Chebyshev, phi=1.0, equilibration=False):
    p = PhysParams()
    p.spring.type = Spring.FENE
    p.spring.sqrtb = 50.0 ** 0.5
    p.hstar, p.hi_method = 0.2, method
    p.ev.type = EV.SDK
    p.ev.dstar = 0.5
    p.ev.phi = np.full(N * N, phi)
    p.equilibration = equilibration
    p.flow = flows.shear(0.5)
    p.number_of_beads = N
    s = SimParams()
    s.dt, s.time_start, s.time_end = 5e-3, 0.0, 1e-2
    step = [SEPARATIONS[i % len(SEPARATIONS)] for i in range(N - 1)]
    R = np.zeros((N, 3))
    R[1:, 0] = np.cumsum(step)
    return p, s, R


@pytest.mark.parametrize("equilibration", [False, True])
@pytest.mark.parametrize("N", [2, 8, 66])
def test_forces(port, N, equilibration):
    p, _, R = sdk_chain(N, equilibration=equilibration)
    got, want = B.total_force(R, p), port.total_force(R, p)
    assert np.max(np.abs(got - want)) <= 1e-12 * max(1.0, float(np.max(np.abs(want))))


@pytest.mark.parametrize("form,N,method", [
    ("plain", 8, DelSMethod.Chebyshev), ("plain", 8, DelSMethod.Cholesky), ("plain", 66, DelSMethod.Cholesky),
    ("mixed", 8, DelSMethod.Chebyshev), ("mixed", 8, DelSMethod.Cholesky)])
def test_steps(port, form, N, method):
    """The pair, block and team kernels, in the forms that run them."""
    p, s, R = sdk_chain(N, method, phi=20.0)
    g = Rng(3)
    got = B.integrate(R, p, s, g, form=form)
    want, st, status, _ = port.integrate(R, p, s, (1, -1, 3))
    assert status == 0 and g.state() == st
    rel = float(np.max(np.abs(got - want)) / max(1.0, float(np.max(np.abs(want)))))
    assert rel <= (1e-10 if form == "plain" else 1e-4)
