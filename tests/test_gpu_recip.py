"""S(k) of every atom (ewald1) against a direct sum, where its two kernels and their remainders change: one atom,
chunks filled exactly and by one more, octets with missing members (a short axis, an odd number
of |n|), few blocks (one k-vector a thread) and many (octets), guests of two species before the framework.

Tolerance: a phase built by kmax recurrence steps is off by at most about 3 kmax roundings per axis, so a sum over
charges q by 9 kmax eps sum|q|."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("natoms, kmax, skew, guests", [
    (1, (3, 3, 3), 0.0, 0),
    (134, (5, 5, 6), 0.0, 0),
    (135, (5, 5, 6), 0.15, 7),
    (300, (4, 1, 7), 0.0, 5),
    (300, (1, 6, 1), 0.1, 0),
    (2000, (8, 9, 7), 0.0, 31),
    (2600, (12, 11, 12), 0.12, 150),
])
def test_structure_factor(fmc, tmp_path, natoms, kmax, skew, guests):
    from fastmc_b200 import synth

    s = max((natoms / 0.025) ** (1.0 / 3.0), 27.0)
    rng = np.random.default_rng(natoms)
    cell = np.array([[s, 0, 0], [skew * s, 1.02 * s, 0], [0, skew * s, 1.05 * s]])
    types = [t for t, _, _ in synth.FRAMEWORK_TYPES]
    names = sorted((types[i % 4] for i in range(natoms)), key=types.index)
    fw = synth.Framework(np.round(cell, 12), names, np.round(rng.uniform(0, 1, (natoms, 3)) @ cell, 12),
                         np.round(rng.normal(0, 0.4, natoms), 10), {t: (0.1, 3.0) for t in types})
    d = synth.write_inputs(str(tmp_path / "deck"), fw, ["CO2", "N2"], [1.0, 1.0], 298.0, kmax)
    c = fmc.Chain(d)
    xyz, q = [fw.xyz], [fw.charges]
    for g, charge in ((0, [0.7, -0.35, -0.35]), (1, [-0.482, 0.964, -0.482])):
        if guests:
            mol = rng.uniform(0, 1, (guests + g, 1, 3)) @ cell + rng.uniform(-1, 1, (guests + g, 3, 3))
            c.set_guests(g, mol)
            xyz.append(mol.reshape(-1, 3))
            q.append(np.tile(charge, guests + g))
    c.ewald1()
    xyz, q = np.concatenate(xyz), np.concatenate(q)
    lmn, _ = c.kvectors()
    frac = xyz @ np.linalg.inv(cell)
    ref = np.concatenate([np.exp(2j * np.pi * (lmn[i:i + 256] @ frac.T)) @ q for i in range(0, len(lmn), 256)])
    eps = np.finfo(float).eps
    # the direct sum's own arguments are off by eps |l x + m y + n z|, at most 3 kmax wraps of a cell
    tol = (9 * max(kmax) + 2 * np.pi * 3 * max(kmax) + len(q)) * eps * np.abs(q).sum() / 2
    assert np.max(np.abs(c.sk() - ref)) <= tol
