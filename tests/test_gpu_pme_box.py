"""A batch whose members' reciprocal sums are done by a block each (FZ_BATCH_BOX=1, the
rule for 8 members or more) against each member alone, on the launches over bricks and
planes: the lines go through the same stages, so states and forces are equal bit for bit,
at every compiled grid size (odd ones among them: a row without a partner), with fewer and
with more atoms than the block has threads, and beside members that keep the launches (a grid
too large, an atom more than a block takes).  The launches of a step say which way it went."""
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


def _path(K, nw, box=24.0):
    return system(f"box_{K}_{nw}", name="custom", nw=nw, nchains=0, box=box, kgrid=K, rc=8.0, ron=6.5, seed=K)[1]


# (grid, waters, box edge) of the members, and how many take a block
@pytest.mark.parametrize("members,blocks", [
    ([(16, 150, 24.0), (18, 150, 24.0), (20, 150, 24.0)], 3),
    ([(24, 400, 24.0), (25, 400, 24.0), (27, 400, 24.0)], 3),
    ([(30, 400, 24.0), (32, 400, 24.0), (36, 400, 24.0)], 3),
    ([(27, 400, 24.0), (40, 400, 24.0), (16, 150, 24.0)], 2),
    ([(32, 2666, 43.1), (36, 2667, 43.1), (24, 400, 24.0)], 2),  # 7,998 and 8,001 atoms
])
def test_members_equal_themselves_alone(members, blocks, monkeypatch):
    paths = [_path(*m) for m in members]
    alone = [_load(p) for p in paths]
    for s in alone:
        s.SingleStep(12)
    launches = {}
    for least in ("1", "1000"):
        monkeypatch.setenv("FZ_BATCH_BOX", least)
        mixed = [_load(p) for p in paths]
        b = fz.Batch(mixed)
        b.step(12)
        launches[least] = b.launches_per_step()
        for a, m in zip(alone, mixed):
            assert np.array_equal(a.positions(), m.positions())
            assert np.array_equal(a.velocities(), m.velocities())
            assert np.array_equal(a.forces_fixed(), m.forces_fixed())
        b.close()
        for s in mixed:
            s.close()
    # by launches: seven and three for every grid size; by blocks: one and those of the rest
    rest = len(members) - blocks
    by_launches = 7 + 3 * len({m[0] for m in members})
    assert launches["1000"] - launches["1"] == by_launches - 1 - (7 + 3 * rest if rest else 0)
    for s in alone:
        s.close()
