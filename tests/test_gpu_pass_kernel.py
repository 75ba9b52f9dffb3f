"""The plain pass kernel's real-space blocks (two candidates a thread in flight, 256 threads a site) where their
remainders change: empty and short lists, lists of more than one trip (dense framework), more guests than
one trip holds, single-site molecules (their own order of summation).  Each replays the oracle move for
move within the per-move bar of the other plain tests."""
import numpy as np
import pytest

from test_gpu_plain import _compare_traces

pytestmark = pytest.mark.gpu

NO_ROTATION = {"insert": 0.3, "delete": 0.3, "displace": 0.4}


@pytest.mark.parametrize("natoms, gas, moves, skew", [
    (5, "CO2", None, 0.0),
    (256, "N2", None, 0.15),
    (1300, "CO2", None, 0.0),
    (1300, "CH4", NO_ROTATION, 0.1),
    (40, "CH4", NO_ROTATION, 0.0),
])
def test_pass_replays_oracle(fmc, oracle_mod, tmp_path, natoms, gas, moves, skew):
    from fastmc_b200 import synth

    L = (26.0, 26.5, 27.5)
    fw = synth.make_framework(L, natoms, seed=natoms)
    if skew:
        fw.cell = fw.cell + np.array([[0, 0, 0], [skew * L[0], 0, 0], [0, skew * L[1], 0]])
    d = synth.write_inputs(str(tmp_path / "deck"), fw, [gas], [20.0], 298.0, (4, 4, 5), moves=moves)
    seed = (7, 11, 13, 17)
    _compare_traces(fmc.Chain(d, seed=seed).run(800), oracle_mod.Chain(d, seed=seed).run(800))


def test_many_guests_single_point_and_trial(fmc, oracle_mod, tmp_path):
    """300 CO2 on a grid (900 guest sites, four trips a block): single point and trial energies."""
    from fastmc_b200 import synth

    fw = synth.make_framework((45.0, 45.0, 45.0), 60, seed=3)
    d = synth.write_inputs(str(tmp_path / "deck"), fw, ["CO2"], [1.0], 298.0, (6, 6, 6))
    rng = np.random.default_rng(2)
    g = np.stack(np.meshgrid(*[np.arange(7) * 6.2 + 1.0] * 3, indexing="ij"), -1).reshape(-1, 3)[:300]
    u = rng.normal(size=(300, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    mols = g[:, None, :] + np.array([0.0, 1.16, -1.16])[None, :, None] * u[:, None, :]
    c, orc = fmc.Chain(d), oracle_mod.Chain(d)
    c.set_guests(0, mols)
    orc.load_guests(0, mols.reshape(-1, 3))
    sp, dlp = c.single_point()
    ref = orc.scalars()
    assert abs(sp - ref["spenergy"]) <= 1e-9 * abs(ref["spenergy"])
    assert abs(dlp - ref["dlpeng"]) <= 1e-9 * abs(ref["dlpeng"])
