"""The batched real-space loop (chunks of 32 candidates, one interleaved erc/vdW table) where its
remainders change: lists shorter than a chunk and empty ones, single-site molecules, orthorhombic and
triclinic cells.  Each replays the oracle move for move within the per-move bar of the other batched
tests."""
import numpy as np
import pytest

from test_gpu_plain import _compare_traces

pytestmark = pytest.mark.gpu

NO_ROTATION = {"insert": 0.3, "delete": 0.3, "displace": 0.4}


@pytest.mark.parametrize("natoms, gas, moves, skew", [
    (5, "CO2", None, 0.0),   # most lists empty or a few entries
    (33, "N2", None, 0.15),  # around one chunk
    (66, "CH4", NO_ROTATION, 0.0),
    (400, "CH4", NO_ROTATION, 0.15),
])
def test_pair_loop_replays_oracle(fmc, oracle_mod, tmp_path, natoms, gas, moves, skew):
    from fastmc_b200 import synth

    L = (27.5, 29.0, 31.0)
    fw = synth.make_framework(L, natoms, seed=natoms)
    if skew:
        fw.cell = fw.cell + np.array([[0, 0, 0], [skew * L[0], 0, 0], [0, skew * L[1], 0]])
    d = synth.write_inputs(str(tmp_path / "deck"), fw, [gas], [5.0], 298.0, (4, 5, 5), moves=moves)
    seeds = [(12, 34, 56, 78), (3, 5, 7, 9)]
    b = fmc.Batch([d, d], seeds)
    tr, _ = b.run(1500, trace=True)
    for i, s in enumerate(seeds):
        _compare_traces(tr[i], oracle_mod.Chain(d, seed=s).run(1500))
