"""Systems of several unit classes (free atoms, X-H, X-H2, X-H3, rigid waters): inside a step
the first half of the classes is integrated on a stream beside the rest.  The classes touch
disjoint atoms, so steps from graphs are bit for bit those launched one after another on one
stream (stage timing), and every constraint holds."""
import dataclasses

import numpy as np
import pytest

import fenzi_b200 as fz
from fenzi_b200 import gen_system

pytestmark = pytest.mark.gpu

# X-H_k molecules, k hydrogens on a tetrahedron's corners, and their parameters
RXH = 1.09
CORNERS = np.array([[1, 1, 1], [1, -1, -1], [-1, 1, -1]]) / np.sqrt(3.0) * RXH
PRM = {"\nANGLES\n": f"CX   HX    340.000   {RXH:.4f}\n\nANGLES\nHX   CX   HX     35.500  109.470\n",
       "\nNBFIX\n": "CX    0.0     -0.1000     1.7500\nHX    0.0     -0.0220     1.3200\n\nNBFIX\n"}


def _write(monkeypatch, outdir, nw, nchains, kinds):
    """nw waters, and one molecule for every entry of kinds (its hydrogens), in place of waters."""
    monkeypatch.setitem(gen_system.TYPES, "CX", (14.027, 0.1, 1.75))
    monkeypatch.setitem(gen_system.TYPES, "HX", (1.008, 0.022, 1.32))
    monkeypatch.setitem(gen_system.RTF_IDS, "CX", 82)
    monkeypatch.setitem(gen_system.RTF_IDS, "HX", 5)
    tot, nch = nw + len(kinds), 10 * nchains
    s = gen_system.build(name="xh", nw=tot, nchains=nchains, chain_len=10, box=(tot * 1.3 / 0.0334) ** (1 / 3), rc=7.0,
                         ron=5.5, seed=tot)
    cut = nch + 3 * nw
    types, names, res, charge, resid, pos = s.types[:cut], s.atom_names[:cut], s.resnames[:cut], list(s.charge[:cut]), \
        list(s.resids[:cut]), list(s.pos[:cut])
    bonds, angles = list(s.bonds[(s.bonds < cut).all(1)]), list(s.angles[(s.angles < cut).all(1)])
    for m, k in enumerate(kinds):
        a, at = len(types), s.pos[cut + 3 * m]
        types += ["CX"] + ["HX"] * k
        names += ["CX"] + [f"HX{j}" for j in range(k)]
        res += [f"XH{k}"] * (k + 1)
        charge += [-0.05 * k] + [0.05] * k
        resid += [nw + m + 1] * (k + 1)
        pos += [at] + [at + CORNERS[j] for j in range(k)]
        bonds += [(a, a + 1 + j) for j in range(k)]
        angles += [(a + 1 + i, a, a + 1 + j) for i in range(k) for j in range(i + 1, k)]
    pos = np.array(pos)
    path = gen_system.write(dataclasses.replace(
        s, pos=pos - np.floor(pos / s.box + 0.5) * s.box, types=types, charge=np.array(charge),
        mass=np.array([gen_system.TYPES[t][0] for t in types]), atom_names=names, resnames=res, segids=["SYS"] * len(types),
        resids=np.array(resid), bonds=np.array(bonds), angles=np.array(angles)), str(outdir))
    prm = outdir / "xh.prm"
    text = prm.read_text()
    for mark, lines in PRM.items():
        assert mark in text
        text = text.replace(mark, lines, 1)
    prm.write_text(text)
    return path


@pytest.mark.parametrize("nw,nchains,kinds", [
    (200, 2, [1, 2, 3] * 20),   # five classes
    (300, 2, [3] * 40),         # three
    (0, 0, [1] * 130 + [2] * 131),  # two, no water
])
def test_classes_beside_one_another_equal_one_after_another(nw, nchains, kinds, monkeypatch, tmp_path):
    path = _write(monkeypatch, tmp_path, nw, nchains, kinds)
    runs = []
    for inline in (False, True):
        s = fz.FenZi.ReadInput(path).LoadSystem()
        s.InitMem(0)
        s.Minimize(200)
        s.InitVelocity(T=50.0, seed=6)
        if inline:
            s.stage_timing(True)
        s.SingleStep(107)  # a chunk graph and seven one-step graphs, or plain launches
        runs.append((s.positions(), s.velocities(), s.forces_fixed()))
        t = s.topology()
        c = t["cons"]
        d = s.positions()[c[:, 0]] - s.positions()[c[:, 1]]
        d -= np.round(d / t["box"]) * t["box"]
        # FP32 coordinates of a box this size: half an ulp of L/2 per coordinate, a few of them
        assert np.abs(np.linalg.norm(d, axis=1) - t["cons_d"]).max() < 4 * np.spacing(np.float32(t["box"][0] / 2))
        s.close()
    for a, b in zip(*runs):
        assert np.array_equal(a, b)
