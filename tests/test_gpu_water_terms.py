"""The forces a step leaves behind against a force call at its positions, bit for bit (all sums
are integers).  In a step the rigid waters' own terms come from the integrator's pass, and PME
and the other bonded terms read the positions before a rebuild wraps them; a force call has
every term from its own kernel and reads the wrapped ones.  Steps that rebuild are among those
compared.  With chains (two unit classes in one launch) and without, around the 32 waters of a
block with four lanes each and the 128 of one with a lane each; the terms themselves are checked
against the oracle in test_gpu_terms.py."""
import numpy as np
import pytest

import fenzi_b200 as fz
from tests.helpers import system

pytestmark = pytest.mark.gpu


def _start(nw, chains, T=300.0, flexible=False):
    kw = {} if chains == 0 else dict(chain_len=10, extras=flexible)
    _, path = system(f"wt_{nw}_{chains}_{flexible}", name="custom", nw=nw, nchains=chains, rc=6.5, ron=5.0, seed=nw, **kw)
    s = fz.FenZi.ReadInput(path)
    s.cfg.shake = 0 if flexible else 1
    s.LoadSystem()
    s.InitMem(0)
    s.InitVelocity(T=T, seed=5)
    return s


@pytest.mark.parametrize("few", ["0", "1000000"], ids=["one_lane", "four_lanes"])
@pytest.mark.parametrize("nw,chains", [(127, 0), (128, 2), (129, 0), (160, 1), (161, 0), (400, 3)])
def test_forces_left_by_a_step_equal_a_force_call(nw, chains, few, monkeypatch):
    monkeypatch.setenv("FZ_FEW_WATERS", few)
    s = _start(nw, chains)
    at_rebuild = 0
    for n in (1, 2, 3) + (1,) * 20:
        s.SingleStep(n - 1)
        before = s.counters()["rebuilds"]
        s.SingleStep(1)
        at_rebuild += s.counters()["rebuilds"] > before
        left = s.forces_fixed()
        s.ComputeAccelGPU()
        assert np.array_equal(left, s.forces_fixed())
    assert at_rebuild >= 2
    s.close()


@pytest.mark.parametrize("nw,chains,kind", [(400, 0, "rigid"), (900, 2, "rigid"), (900, 2, "flexible"), (900, 2, "barostat")])
def test_a_run_does_not_depend_on_its_print_interval(nw, chains, kind):
    """flexible: every bonded term (Urey-Bradley, impropers, two folds) and no constraint."""
    a, b = (_start(nw, chains, flexible=kind == "flexible") for _ in range(2))
    if kind == "barostat":
        for s in (a, b):
            s.set_barostat(True, pref_atm=1.0, pmass=1e-5)
    for k in range(40):
        a.SingleStep(3)
        b.SingleStep(3)
        b.EvalProps()
    assert b.counters()["rebuilds"] > 10
    assert np.array_equal(a.positions(), b.positions())
    assert np.array_equal(a.velocities(), b.velocities())
    for s in (a, b):
        s.close()


@pytest.mark.parametrize("npt", [False, True], ids=["chunk_graph", "barostat"])
@pytest.mark.parametrize("nw,chains", [(127, 0), (129, 2), (400, 3)])
def test_one_lane_a_water_equals_four(nw, chains, npt, monkeypatch):
    """Every form of the pass: alone, beside free atoms, closing the step before, under the
    barostat."""
    runs = []
    for few in ("0", "1000000"):
        monkeypatch.setenv("FZ_FEW_WATERS", few)
        s = _start(nw, chains)
        if npt:
            s.set_barostat(True, pref_atm=1.0, pmass=1e-5)
        s.SingleStep(20 if npt else 107)
        runs.append((s.positions(), s.velocities(), s.forces_fixed()))
        s.close()
    for a, b in zip(*runs):
        assert np.array_equal(a, b)


def test_the_line_between_one_lane_and_four(monkeypatch):
    """A system of as many waters as the line and one of one more: the two sides of the rule."""
    for few in ("400", "399"):
        monkeypatch.setenv("FZ_FEW_WATERS", few)
        s = _start(400, 3)
        s.SingleStep(25)
        if few == "400":
            want = s.positions()
        else:
            assert np.array_equal(want, s.positions())
        s.close()
