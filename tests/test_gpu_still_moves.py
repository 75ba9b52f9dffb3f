"""Moves that leave their molecule in place: a single site's rotation, a rotation whose angle is drawn as exactly
zero (draws are multiples of 2^-24), a translation with no step size.

Their energy change is the rounding of two equal sums, and its sign decides whether the acceptance test draws a
random number (gcmc.f:1330-1338), so a seeded chain repeats only if these sums keep every bit.  The oracle rounds
differently, so the values are those recorded in golden/still_moves.json with the library of commit f22ff4d: the
energies of every such move and the reciprocal energy of every move (which carries S(k)) bit for bit, and every
decision.  `python tests/test_gpu_still_moves.py OUT` records them with the library found on PYTHONPATH."""
import hashlib
import json
import os
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
pytestmark = pytest.mark.gpu

BOX = (27.5, 29.0, 31.0)
ION = ("ION", [("Kx", 39.098, 0.8, 0.0, 0.0, 0.0, 0.1, 3.1)])  # a charged single site
TURN = {"insert": 0.2, "rotate": 0.8}
STEP = {"insert": 0.3, "delete": 0.1, "translate": 0.6}
MANY = {"insert": 0.25, "delete": 0.15, "displace": 0.2, "rotate": 0.4}

# name: (cell, framework atoms, gases, moves, step size, seed, number of moves)
CASES = {
    # seeds whose zero angle comes within a few hundred draws
    "zero_angle_co2": ("ortho", 66, ["CO2"], TURN, 1.0, (85, 163, 1, 48), 220),
    "zero_angle_co2_cubic": ("cubic", 90, ["CO2"], TURN, 1.0, (163, 68, 32, 155), 120),
    "zero_angle_n2": ("triclinic", 80, ["N2"], TURN, 1.0, (138, 106, 136, 24), 200),
    "zero_angle_n2_late": ("triclinic", 80, ["N2"], TURN, 1.0, (39, 68, 28, 110), 220),
    "zero_angle_mixture": ("triclinic", 70, ["CO2", "N2"], TURN, 1.0, (54, 102, 135, 44), 100),
    # every translation stays in place
    "no_step_co2": ("ortho", 66, ["CO2"], STEP, 0.0, (3, 5, 7, 9), 400),
    "no_step_n2": ("cubic", 300, ["N2"], STEP, 0.0, (12, 34, 56, 78), 400),
    "no_step_mixture": ("triclinic", 70, ["CO2", "N2"], STEP, 0.0, (11, 13, 17, 19), 400),
    "no_step_empty": ("ortho", 5, ["CO2"], STEP, 0.0, (3, 5, 7, 11), 300),
    "no_step_octahedron": ("imcon4", 0, ["CO2"], STEP, 0.0, (3, 5, 7, 13), 200),
    "no_step_dodecahedron": ("imcon5", 0, ["N2"], STEP, 0.0, (3, 5, 7, 27), 200),
    "no_step_prism": ("imcon7", 0, ["CO2"], STEP, 0.0, (3, 5, 7, 29), 200),
    "no_step_slab": ("imcon6", 0, ["N2"], STEP, 0.0, (3, 5, 7, 15), 200),
    "no_step_tilted_slab": ("tilted", 0, ["CO2"], STEP, 0.0, (3, 5, 7, 31), 200),
    "no_step_rvdw": ("rvdw", 66, ["CO2"], STEP, 0.0, (3, 5, 7, 17), 200),
    # every rotation of a single site
    "ch4": ("ortho", 66, ["CH4"], MANY, 1.0, (3, 5, 7, 9), 600),
    "ch4_few_atoms": ("triclinic", 5, ["CH4"], MANY, 1.0, (3, 5, 7, 21), 400),
    "ch4_n2": ("triclinic", 400, ["CH4", "N2"], MANY, 1.0, (3, 5, 7, 23), 600),
    "ion": ("ortho", 66, [ION], MANY, 1.0, (3, 5, 7, 25), 400),
}


def deck(synth, root, name):
    cell, natoms, gases, moves, delr, _, _ = CASES[name]
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
    d = synth.write_inputs(os.path.join(str(root), name), fw, gases, [50.0] * len(gases), 298.0, kmax, moves=moves,
                           delr=delr, imcon=imcon)
    if cell == "rvdw":  # tables of two spacings
        path = os.path.join(d, "CONTROL")
        text = open(path).read().replace("finish", "rvdw cutoff 13.500000\nfinish")
        open(path, "w").write(text)
    return d


def trace(fmc, d, name, path):
    """The traces of the case's chain: two chains of a batch, or the plain chain."""
    seed, n = CASES[name][5:]
    if path == "plain":
        return [fmc.Chain(d, seed=seed).run(n)]
    b = fmc.Batch([d, d], [seed, tuple(seed[:3]) + (2,)])
    return list(b.run(n, trace=True)[0])


def still(t, name):
    """Which moves of a trace leave their molecule in place (found by their energy change)."""
    return (t["mtype"] >= 3) & (t["mtype"] <= 5) & (np.abs(t["estep"]) < 1e-9)


def digest(a):
    return hashlib.sha256(np.ascontiguousarray(a).tobytes()).hexdigest()[:24]


def summary(t, name):
    s = still(t, name)
    return {"still": int(s.sum()),
            "decisions": digest(np.stack([t[k] for k in ("iguest", "mtype", "randchoice", "accepted", "nmols_after")])),
            "draws": digest(t["rande"]),
            "recip": digest(t["ewld1"]),
            "ewld2": digest(t["ewld2"][s]), "vdw": digest(t["vdw"][s]), "estep": digest(t["estep"][s])}


def record(fmc, synth, root):
    out = {}
    for name in CASES:
        d = deck(synth, root, name)
        for path in ("batched", "plain"):
            out["%s/%s" % (name, path)] = [summary(t, name) for t in trace(fmc, d, name, path)]
    return out


@pytest.fixture(scope="module")
def golden():
    with open(os.path.join(HERE, "golden", "still_moves.json")) as f:
        return json.load(f)


@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("path", ["batched", "plain"])
def test_still_moves_keep_their_bits(fmc, tmp_path, golden, name, path):
    from fastmc_b200 import synth

    got = [summary(t, name) for t in trace(fmc, deck(synth, tmp_path, name), name, path)]
    want = golden["%s/%s" % (name, path)]
    assert want[0]["still"] > 0
    assert got == want


if __name__ == "__main__":
    import tempfile

    import fastmc_b200
    from fastmc_b200 import synth as _synth

    with open(sys.argv[1], "w") as _f:
        json.dump(record(fastmc_b200, _synth, tempfile.mkdtemp()), _f, indent=1)
