"""Real-space energies of the plain pass (ewald2 + srfrce) and the sums over all atoms, bit for bit.

A host move loop over the drop-in calls decides a move that leaves its molecule in place (an angle drawn as exactly
zero) by what these sums round off: E_new < E_old takes no draw (gcmc.f:1330-1338).  So a seeded loop repeats only
if every energy keeps its bits.  The oracle rounds differently; the values are those recorded in
golden/dropin_bits.json with the library of commit f22ff4d: energies of molecules in place, displaced and inserted,
with and without an update left pending by a commit, every energy of a plain run, ewald1 and single_point.
`python tests/test_gpu_dropin_bits.py OUT` records them with the library found on PYTHONPATH."""
import hashlib
import json
import os
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
pytestmark = pytest.mark.gpu

BOX = (27.5, 29.0, 31.0)
# name: (cell, framework atoms, gases, guests of each, moves of the run)
CASES = {
    "ortho_co2": ("ortho", 700, ["CO2"], 40, 300),
    "ortho_few_atoms": ("ortho", 5, ["CO2"], 3, 200),
    "ortho_many_guests": ("ortho", 66, ["CO2"], 180, 100),
    "ortho_ch4": ("ortho", 500, ["CH4"], 30, 300),
    "cubic_n2": ("cubic", 600, ["N2"], 25, 300),
    "triclinic_co2": ("triclinic", 600, ["CO2"], 40, 300),
    "triclinic_mixture": ("triclinic", 300, ["CO2", "N2"], 20, 300),
    "triclinic_ch4": ("triclinic", 300, ["CH4"], 20, 200),
    "octahedron": ("imcon4", 0, ["CO2"], 10, 200),
    "dodecahedron": ("imcon5", 0, ["N2"], 10, 200),
    "prism": ("imcon7", 0, ["CO2"], 10, 200),
    "slab": ("imcon6", 0, ["N2"], 10, 200),
    "tilted_slab": ("tilted", 0, ["CO2"], 10, 200),
    "rvdw": ("rvdw", 300, ["CO2"], 20, 200),
    "rvdw_ch4": ("rvdw", 300, ["CH4"], 20, 200),
    "many_k": ("ortho", 1500, ["CO2"], 60, 100),
    "many_k_triclinic": ("triclinic", 200, ["CO2", "N2"], 60, 100),
}


def deck(synth, root, name):
    cell, natoms, gases, _, _ = CASES[name]
    imcon, kmax = None, (4, 5, 5)
    if cell in ("imcon4", "imcon5", "imcon7"):
        imcon = int(cell[5:])
        fw = synth.half_shift_framework(imcon, 30.0, seed=40 + imcon)
    elif cell in ("imcon6", "tilted"):
        imcon, kmax, fw = 6, (4, 4, 9), synth.slab_framework(28.0, 20.0, 60.0, seed=46)
        if cell == "tilted":
            fw.cell[1, 0] = 5.0
    else:
        fw = synth.make_framework((28.0,) * 3 if cell == "cubic" else BOX, natoms, seed=natoms)
        if cell == "triclinic":
            fw.cell = fw.cell + np.array([[0, 0, 0], [0.15 * BOX[0], 0, 0], [0, 0.15 * BOX[1], 0]])
    if name.startswith("many_k"):
        kmax = (12, 12, 13)
    d = synth.write_inputs(os.path.join(str(root), name), fw, gases, [20.0] * len(gases), 298.0, kmax, imcon=imcon)
    if cell == "rvdw":  # tables of two spacings
        path = os.path.join(d, "CONTROL")
        text = open(path).read().replace("finish", "rvdw cutoff 13.500000\nfinish")
        open(path, "w").write(text)
    return d, fw


def molecules(synth, rng, gas, fw, n):
    """n molecules anywhere in the cell (energies need not be physical, only finite)."""
    site = np.array([s[3:6] for s in synth.GASES[gas][1]])[:, :1]
    u = rng.normal(size=(n, 1, 3))
    u /= np.linalg.norm(u, axis=2)[:, :, None]
    return rng.uniform(0.02, 0.98, (n, 1, 3)) @ fw.cell + site[None] * u


def values(fmc, synth, root, name):
    """Energies of the drop-in calls, as hexadecimal numbers, and digests of a run's energies."""
    _, _, gases, guests, moves = CASES[name]
    d, fw = deck(synth, root, name)
    rng = np.random.default_rng(len(name))
    c = fmc.Chain(d, seed=(3, 5, 7, 9))
    out = []
    for g, gas in enumerate(gases):
        mols = molecules(synth, rng, gas, fw, guests + 6)
        c.set_guests(g, mols[:guests])
        for k in range(3):
            mol = int(rng.integers(0, guests))
            out += c.guest_realspace(g, mols[mol], mol)  # in place
            out += c.guest_realspace(g, mols[mol] + rng.uniform(-0.3, 0.3, 3), mol)
            out += c.guest_realspace(g, mols[guests + k])
        # an insertion and a deletion whose updates the next call reads through
        c.ewald1_guest(g, mols[guests + 4], fmc.INSERT)
        c.commit(fmc.INSERT, g, -1, mols[guests + 4])
        out += c.guest_realspace(g, mols[guests + 5])
        c.ewald1_guest(g, mols[1], fmc.DELETE)
        c.commit(fmc.DELETE, g, 1)
        out += c.guest_realspace(g, mols[0], 0)
        out += c.guest_realspace(g, mols[2] + 1e-9, 1)
    sums = [c.ewald1(), *c.single_point()]
    assert np.all(np.isfinite(out + sums))
    t = fmc.Chain(d, seed=(3, 5, 7, 11)).run(moves)
    return {"calls": [float(v).hex() for v in out], "sums": [float(v).hex() for v in sums],
            **{k: hashlib.sha256(np.ascontiguousarray(t[k]).tobytes()).hexdigest()[:24]
               for k in ("mtype", "accepted", "ewld1", "ewld2", "vdw", "estep")}}


@pytest.fixture(scope="module")
def golden():
    with open(os.path.join(HERE, "golden", "dropin_bits.json")) as f:
        return json.load(f)


@pytest.mark.parametrize("name", CASES)
def test_real_space_keeps_its_bits(fmc, tmp_path, golden, name):
    from fastmc_b200 import synth

    assert values(fmc, synth, tmp_path, name) == golden[name]


if __name__ == "__main__":
    import tempfile

    import fastmc_b200
    from fastmc_b200 import synth as _synth

    with open(sys.argv[1], "w") as _f:
        json.dump({n: values(fastmc_b200, _synth, tempfile.mkdtemp(), n) for n in CASES}, _f, indent=1)
