"""Batched ensemble: every system gives the same result alone and in the batch."""
import os
import tempfile

import numpy as np
import pytest

import fenzi_b200 as fz
from fenzi_b200 import gen_system

pytestmark = pytest.mark.gpu


def _load(s, d):
    p = gen_system.write(s, d)
    sy = fz.FenZi.ReadInput(p).LoadSystem()
    sy.InitMem(0)
    sy.InitVelocity(T=300.0, seed=77)
    return sy


def test_batch_matches_each_system_alone():
    systems = gen_system.ensemble(nsys=5, seed=11, nw_min=216, nw_max=700)
    tmp = tempfile.mkdtemp(prefix="fzbatch_")
    alone = [_load(s, os.path.join(tmp, f"a{i}")) for i, s in enumerate(systems)]
    mixed = [_load(s, os.path.join(tmp, f"b{i}")) for i, s in enumerate(systems)]
    for s in alone:
        s.SingleStep(25)
    b = fz.Batch(mixed)
    b.step(25)
    for a, m in zip(alone, mixed):
        assert np.array_equal(a.positions(), m.positions())
        assert np.array_equal(a.velocities(), m.velocities())
        assert np.array_equal(a.forces_fixed(), m.forces_fixed())
    b.close()
    for s in alone + mixed:
        s.close()


def test_batched_kernels_match_per_system_branches():
    """The batched kernels (one launch per kernel over all members) and the graph of
    per-member branches give bit-identical trajectories, on members with chains (free-
    atom and bonded-term classes besides rigid water) and odd grid sizes (25, 27)."""
    specs = [dict(nw=300, nchains=2, chain_len=10, box=24.0, kgrid=25),
             dict(nw=420, nchains=0, box=25.5, kgrid=27),
             dict(nw=260, nchains=1, chain_len=12, box=22.0, kgrid=24),
             dict(nw=500, nchains=3, chain_len=8, box=27.0, kgrid=32)]
    tmp = tempfile.mkdtemp(prefix="fzbk_")
    runs = {}
    for mode in ("1", "0"):
        old = os.environ.get("FZ_BATCH_KERNELS")
        os.environ["FZ_BATCH_KERNELS"] = mode
        try:
            sys_ = [_load(gen_system.build(name="custom", rc=9.0, ron=7.5, seed=40 + i, **sp),
                          os.path.join(tmp, f"{mode}_{i}")) for i, sp in enumerate(specs)]
            b = fz.Batch(sys_)
            b.step(30)
            runs[mode] = [(s.positions(), s.velocities(), s.forces_fixed()) for s in sys_]
            b.close()
            for s in sys_:
                s.close()
        finally:
            if old is None:
                os.environ.pop("FZ_BATCH_KERNELS", None)
            else:
                os.environ["FZ_BATCH_KERNELS"] = old
    for (p1, v1, f1), (p0, v0, f0) in zip(runs["1"], runs["0"]):
        assert np.array_equal(p1, p0)
        assert np.array_equal(v1, v0)
        assert np.array_equal(f1, f0)


@pytest.mark.parametrize("kernels", ["1", "0"])
@pytest.mark.parametrize("how", ["state", "positions", "checkpoint"])
def test_members_given_new_positions_start_from_their_forces(how, kernels, monkeypatch, tmp_path):
    """New positions for members of a batch that has already stepped: the next step opens
    with the forces of those positions, as a system alone does (bit for bit)."""
    monkeypatch.setenv("FZ_BATCH_KERNELS", kernels)
    systems = gen_system.ensemble(nsys=3, seed=23, nw_min=216, nw_max=400)
    alone = [_load(s, str(tmp_path / f"a{i}")) for i, s in enumerate(systems)]
    mixed = [_load(s, str(tmp_path / f"b{i}")) for i, s in enumerate(systems)]
    start = [(s.positions(), s.velocities()) for s in alone]
    alone[0].SaveCheckpoint(str(tmp_path / "r"), "b")
    b = fz.Batch(mixed)
    b.step(7)
    for s in alone:
        s.SingleStep(7)
    for i in (0, 2):  # the other member goes on
        for s in (alone[i], mixed[i]):
            if how == "checkpoint" and i == 0:
                s.LoadCheckpoint(str(tmp_path / "r"), "b")
            elif how == "positions":
                s.set_positions(start[i][0])
            else:
                s.set_state_f32(start[i][0].astype(np.float32), start[i][1].astype(np.float32))
    b.step(5)
    for a, m in zip(alone, mixed):
        a.SingleStep(5)
        assert np.array_equal(a.positions(), m.positions())
        assert np.array_equal(a.velocities(), m.velocities())
        assert np.array_equal(a.forces_fixed(), m.forces_fixed())
    b.close()
    for s in alone + mixed:
        s.close()


@pytest.mark.parametrize("kernels", ["1", "0"])
def test_batch_follows_members_of_another_box_or_uploaded_anew(kernels, monkeypatch, tmp_path):
    """The graph of a batch holds its members' boxes and device addresses.  A restart file of
    another box and a new upload change them between two calls: the members still move as
    they do alone, bit for bit."""
    monkeypatch.setenv("FZ_BATCH_KERNELS", kernels)
    systems = gen_system.ensemble(nsys=3, seed=31, nw_min=400, nw_max=500)
    piston = _load(systems[0], str(tmp_path / "p"))
    piston.set_barostat(True, pref_atm=1.0, pmass=1e-6)
    piston.SingleStep(20)
    piston.SaveCheckpoint(str(tmp_path / "r"), "b")
    assert abs(piston.EvalProps()["box"][0] / systems[0].box[0] - 1.0) > 1e-5
    alone = [_load(s, str(tmp_path / f"a{i}")) for i, s in enumerate(systems)]
    mixed = [_load(s, str(tmp_path / f"b{i}")) for i, s in enumerate(systems)]
    b = fz.Batch(mixed)
    b.step(6)
    for s in alone:
        s.SingleStep(6)
    for s in (alone[0], mixed[0]):
        s.LoadCheckpoint(str(tmp_path / "r"), "b")
    for s in (alone[1], mixed[1]):
        s.InitMem(0)
        s.InitVelocity(T=200.0, seed=4)
    b.step(6)
    for a, m in zip(alone, mixed):
        a.SingleStep(6)
        assert np.array_equal(a.positions(), m.positions())
        assert np.array_equal(a.velocities(), m.velocities())
    b.close()
    for s in alone + mixed + [piston]:
        s.close()


def test_members_of_many_columns_take_the_batched_kernels(monkeypatch, tmp_path):
    """A wide flat box has more sorting columns (here 65 x 65) than a block scans in shared
    memory; the batch scans that member's by a launch of its own and keeps its kernels for
    all members, which move as they do alone."""
    monkeypatch.setenv("FZ_COL_ATOMS", "8")
    flat = gen_system.build(name="flat", nw=6000, kgrid=64, rc=5.0, ron=4.0, seed=8)
    own = flat.pos.reshape(-1, 3, 3) - flat.pos.reshape(-1, 3, 3)[:, :1]
    own -= np.round(own / flat.box) * flat.box
    flat.box = np.array([1400.0, 1400.0, 11.5])
    k = np.arange(6000)
    site = np.stack([(k % 78 + 0.5) / 78 * 1400 - 700, (k // 78 + 0.5) / 78 * 1400 - 700, np.zeros(6000)], 1)
    flat.pos = (site[:, None] + own).reshape(-1, 3)
    specs = [gen_system.ensemble(nsys=1, seed=3, nw_min=300, nw_max=300)[0], flat]
    alone = [_load(s, str(tmp_path / f"a{i}")) for i, s in enumerate(specs)]
    for s in alone:
        s.SingleStep(15)
    launches = {}
    for mode in ("1", "0"):
        monkeypatch.setenv("FZ_BATCH_KERNELS", mode)
        mixed = [_load(s, str(tmp_path / f"b{mode}{i}")) for i, s in enumerate(specs)]
        b = fz.Batch(mixed)
        b.step(15)
        launches[mode] = b.launches_per_step()
        for a, m in zip(alone, mixed):
            assert np.array_equal(a.positions(), m.positions())
            assert np.array_equal(a.forces_fixed(), m.forces_fixed())
        b.close()
        for s in mixed:
            s.close()
    assert launches["1"] < launches["0"]
    for s in alone:
        s.close()
