"""Voxel lists where the float test of an orthorhombic cell decides least.

The lists are the atoms within a limit of a voxel's centre (the reference gathers them per trial in
guestlistgen, utility_pack.f:3113-3177); the host's lists take every distance in double, and the device's
must equal them entry for entry.  Atoms are put a millionth of an angstrom inside the limiting sphere of
many voxels, thousands of times closer than the float test can tell, and on the borders between two images; the cell sizes and atom counts leave remainders of the
kernel's groups of voxels and atoms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("edge", [2.0, 1.3])
@pytest.mark.parametrize("lengths", [(25.3, 25.3, 25.3), (25.2, 31.7, 60.9)])
@pytest.mark.parametrize("far", [0.0, 40.0])
def test_atoms_on_the_limit(fmc, tmp_path, lengths, edge, far):
    from fastmc_b200 import synth

    L = np.array(lengths)
    rng = np.random.default_rng(7)
    n = np.maximum(np.floor(L / edge).astype(int), 1)
    w = L / n
    limit = 12.5 + 0.5 * np.linalg.norm(w)  # cut-off and the voxel's circumradius; the lists reach 1e-6 further
    centre = (rng.integers(0, n, (600, 3)) + 0.5) * w
    u = rng.normal(size=(600, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    shell = centre + u * (limit * (1.0 + rng.integers(-3, 4, 600) * 1e-9))[:, None]
    border = centre + rng.choice([-0.5, 0.5], (100, 3)).repeat(6, 0) * L  # half a period off on each axis
    inside = rng.uniform(0.0, 1.0, (37, 3)) * L
    xyz = np.concatenate([shell, border, inside])
    xyz[::3] += far * L  # places given many periods away
    fw = synth.batched_frameworks(2, seed=5)[1]
    k = rng.integers(0, len(fw.names), len(xyz))
    fw = type(fw)(np.diag(L), [fw.names[i] for i in k], xyz, np.zeros(len(xyz)), fw.lj)
    d = synth.write_inputs(str(tmp_path / "d"), fw, ["CO2"], [1.0], 298.0, (2, 2, 2))
    b = fmc.Batch([d], [(1, 2, 3, 4)], voxel_edge=edge)
    nv, off, at = b.voxels(0)
    nv_h, off_h, at_h = fmc.deck_voxels(d, edge)
    assert nv == nv_h
    assert np.array_equal(off, off_h)
    assert np.array_equal(at, at_h)
