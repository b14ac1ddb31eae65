"""The rigid waters' own terms, evaluated by the integrator's pass in a step and by the
bonded kernel in a force call: the forces a step leaves behind are those of a force call
at its positions, bit for bit (all sums are integers), as long as the last step has not
wrapped positions (no rebuild).  Unit counts around a 128-thread block, with chains (two
unit classes in one launch) and without; the terms themselves are checked against the
oracle in test_gpu_terms.py."""
import numpy as np
import pytest

import fenzi_b200 as fz
from tests.helpers import system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nw,chains", [(127, 0), (128, 2), (129, 0), (400, 3)])
def test_forces_left_by_a_step_equal_a_force_call(nw, chains):
    kw = {} if chains == 0 else dict(chain_len=10)
    _, path = system(f"wt_{nw}_{chains}", name="custom", nw=nw, nchains=chains, rc=6.5, ron=5.0, seed=nw, **kw)
    s = fz.FenZi.ReadInput(path).LoadSystem()
    s.InitMem(0)
    s.InitVelocity(T=100.0, seed=5)
    s.SingleStep(1)  # the list rebuild of the start
    for n in (1, 2, 3):
        before = s.counters()["rebuilds"]
        s.SingleStep(n)
        left = s.forces_fixed()
        s.ComputeAccelGPU()
        if s.counters()["rebuilds"] == before:
            assert np.array_equal(left, s.forces_fixed())
    assert s.counters()["rebuilds"] < 4
    s.close()
