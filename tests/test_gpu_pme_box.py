"""A batch whose members' reciprocal sums are done by a block each (FZ_BATCH_BOX=1, the
rule for 8 members or more) against each member alone, on the launches over bricks and
planes: the lines go through the same stages, so states and forces are equal bit for bit,
at every compiled grid size (odd ones among them: a row without a partner), with fewer and
with more atoms than the block has threads, and beside a member whose grid is too large."""
import os

import numpy as np
import pytest

import fenzi_b200 as fz
from tests.helpers import system

pytestmark = pytest.mark.gpu


def _load(path):
    s = fz.FenZi.ReadInput(path).LoadSystem()
    s.InitMem(0)
    s.InitVelocity(T=300.0, seed=9)
    return s


@pytest.mark.parametrize("sizes", [(16, 18, 20), (24, 25, 27), (30, 32, 36), (27, 40, 16)])
def test_members_equal_themselves_alone(sizes):
    paths = [system(f"box_{K}", name="custom", nw=150 if K < 24 else 400, nchains=0, box=24.0, kgrid=K, rc=8.0, ron=6.5,
                    seed=K)[1] for K in sizes]
    alone, mixed = [_load(p) for p in paths], [_load(p) for p in paths]
    for s in alone:
        s.SingleStep(12)
    os.environ["FZ_BATCH_BOX"] = "1"
    try:
        b = fz.Batch(mixed)
        b.step(12)
    finally:
        os.environ.pop("FZ_BATCH_BOX", None)
    for a, m in zip(alone, mixed):
        assert np.array_equal(a.positions(), m.positions())
        assert np.array_equal(a.velocities(), m.velocities())
        assert np.array_equal(a.forces_fixed(), m.forces_fixed())
    b.close()
    for s in alone + mixed:
        s.close()
