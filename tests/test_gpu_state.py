"""State transfer through packed FP32 triples and the forces handed to the host, at atom
counts on both sides of a 256-thread block and at 100,203 atoms.  Exact: every value is a
copy or a power-of-two scaling."""
import numpy as np
import pytest

import fenzi_b200 as fz
from tests.helpers import system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nw", [85, 256, 341, 33401])
def test_packed_state_and_forces_are_exact(nw):
    big = nw > 1000
    _, path = system(f"state_{nw}", name="custom", nw=nw, nchains=0, rc=9.0 if big else 6.0, ron=7.5 if big else 5.0, seed=nw)
    s = fz.FenZi.ReadInput(path).LoadSystem()
    s.InitMem(0)
    n = s.n
    rng = np.random.default_rng(nw)
    L = np.array(list(s.cfg.box))
    pos = s.positions().astype(np.float32) + rng.normal(scale=0.01, size=(n, 3)).astype(np.float32)
    vel = rng.normal(size=(n, 3)).astype(np.float32)
    s.set_state_f32(pos, None)
    s.set_state_f32(None, vel)
    p, v = np.empty((n, 3), np.float32), np.empty((n, 3), np.float32)
    s.get_state_f32(p, v)
    assert np.array_equal(p, pos) and np.array_equal(v, vel)
    s.ComputeAccelGPU()  # charges kept: the oracle-checked forces of these positions
    f, fx = s.forces(), s.forces_fixed().reshape(3, n).T
    assert np.array_equal(f, fx.astype(np.float64) / 2.0 ** 32)
    s.set_positions(pos.astype(np.float64))
    s.ComputeAccelGPU()
    assert np.array_equal(s.forces_fixed().reshape(3, n).T, fx)
    assert np.abs(s.positions() - pos - L * np.round((s.positions() - pos) / L)).max() < 1e-5
    assert np.array_equal(s.velocities().astype(np.float32), vel)
    s.close()
