"""The two kernels of the full S(k) (ewald1): one k-vector a thread, and eight from one read of the phases (octets),
taken where their blocks number the SMs at least.  Both give the same bits, which a seeded chain relies on when
it restarts from S(k) of its state.  The octets' remainders: one atom, a chunk filled exactly and by one more, fewer
octets than a block, axes so short that octets miss most members (in cells as anisotropic as their kmax, so that
the cut-off leaves every axis its k-vectors).

Tolerance against a direct sum: a phase built by kmax recurrence steps is off by at most about 3 kmax roundings per
axis, so a sum over charges q by 9 kmax eps sum|q|."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ANISO = [(2, 6, 30), (30, 2, 6), (6, 30, 2), (1, 12, 31)]


def _framework(kmax, natoms, charged, skew=0.0):
    """natoms atoms, the first `charged` of them with charges, in a cell whose edges go with kmax."""
    from fastmc_b200 import synth

    rng = np.random.default_rng(sum(kmax))
    L = 8.5 * np.array(kmax) / min(kmax)
    cell = np.round(np.diag(L) + skew * np.array([[0, 0, 0], [L[0], 0, 0], [0, L[1], 0]]), 12)
    frac = rng.uniform(0, 1, (max(natoms, 40000), 3))[:natoms]
    q = np.round(rng.normal(0, 0.4, max(natoms, 40000)), 10)[:natoms]
    q[charged:] = 0.0
    return synth.Framework(cell, ["C"] * natoms, np.round(frac @ cell, 12), q, {"C": (0.1, 3.0)})


def _chain(fmc, root, fw, kmax):
    from fastmc_b200 import synth

    return fmc.Chain(synth.write_inputs(str(root), fw, ["CO2"], [1.0], 298.0, kmax, rcut=4.0, alpha=0.6))


def _chunk(kmax):
    """Atoms of a chunk: their phase tables fill 40 KB, at most 256."""
    return min(256, 40 * 1024 // ((sum(kmax) + 3) * 16))


def _octets(lmn, natoms, kmax):
    """Whether these sizes take the octet kernel."""
    quads = {}
    for l, m, n in np.unique(np.abs(lmn), axis=0):
        quads[l, m] = quads.get((l, m), 0) + 1
    noct = sum((v + 1) // 2 for v in quads.values())
    blocks = (noct + 127) // 128 * -(-natoms // _chunk(kmax))
    return noct, blocks >= torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("kmax, natoms, skew", [
    ((42, 42, 42), 1, 0.0),
    ((42, 42, 42), _chunk((42, 42, 42)), 0.1),
    ((42, 42, 42), _chunk((42, 42, 42)) + 1, 0.0),
    ((3, 3, 3), 148 * _chunk((3, 3, 3)), 0.0),
    ((3, 3, 3), 148 * _chunk((3, 3, 3)) + 1, 0.1),
    *((k, 148 * _chunk(k) + 7, 0.1 * (i % 2)) for i, k in enumerate(ANISO)),
])
def test_octets_against_a_direct_sum(fmc, tmp_path, kmax, natoms, skew):
    fw = _framework(kmax, natoms, natoms, skew)
    c = _chain(fmc, tmp_path / "d", fw, kmax)
    lmn, _ = c.kvectors()
    noct, octets = _octets(lmn, natoms, kmax)
    assert octets
    if not skew:  # a sheared cell's reciprocal widths leave some axes a little less
        assert all(np.abs(lmn[:, a]).max() == kmax[a] for a in range(3))
    if kmax == (3, 3, 3):
        assert noct < 128
    c.ewald1()
    frac = torch.tensor(fw.xyz @ np.linalg.inv(fw.cell), device="cuda")
    q = torch.tensor(fw.charges, device="cuda")
    k = torch.tensor(lmn, dtype=torch.float64, device="cuda")
    ref = torch.zeros(len(k), dtype=torch.complex128, device="cuda")
    for a in range(0, natoms, 512):
        t = k @ frac[a:a + 512].T
        t = 2.0 * np.pi * (t - torch.round(t))
        ref += (torch.complex(torch.cos(t), torch.sin(t)) * q[a:a + 512]).sum(1)
    tol = (9 * max(kmax) + 2 * np.pi * 3 * max(kmax) + natoms) * np.finfo(float).eps * np.abs(fw.charges).sum() / 2
    assert np.max(np.abs(c.sk() - ref.cpu().numpy())) <= tol


@pytest.mark.parametrize("kmax", [(3, 3, 3), (8, 9, 7), *ANISO])
@pytest.mark.parametrize("skew", [0.0, 0.1])
def test_both_kernels_give_the_same_bits(fmc, tmp_path, kmax, skew):
    """A chunk of charged atoms alone, and followed by enough neutral ones that octets are taken: their terms are
    zero."""
    n = _chunk(kmax)
    few = _chain(fmc, tmp_path / "few", _framework(kmax, n, n, skew), kmax)
    many = _chain(fmc, tmp_path / "many", _framework(kmax, 148 * n, n, skew), kmax)
    lmn, _ = few.kvectors()
    assert not _octets(lmn, n, kmax)[1] and _octets(lmn, 148 * n, kmax)[1]
    few.ewald1()
    many.ewald1()
    assert np.array_equal(few.sk(), many.sk())
