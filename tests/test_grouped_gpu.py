"""The grouped class kernels (eri_group.cuh) against the oracle: every fused
class they serve, forced on for small molecules, where every quartet is near,
and for molecules so far apart that most are far."""
import numpy as np
import pytest

import oracle as O
from conftest import load_golden
from hartreefock_b200 import engine as E
from hartreefock_b200 import molecules
from hartreefock_b200.basis_io import basis_path

pytestmark = pytest.mark.gpu


def _spread(distance):
    """Two oxygens and a water, `distance` bohr apart."""
    Z, xyz = molecules.H2O_README
    return [8, 8] + list(Z), np.concatenate([[[0.0, 0.0, 0.0], [0.3, -0.2, 2.3]], xyz + [0.1, distance, 0.7 * distance]])


MOLECULES = {"o2": ([8, 8], np.array([[0.0, 0.0, 0.0], [0.3, -0.2, 2.3]])), "spread6": _spread(6.0),
             "spread40": _spread(40.0), "alkane3": molecules.alkane(3), "oh": molecules.hydroxyl()}


def _density(n, seed):
    A = np.random.default_rng(seed).normal(size=(n, n)) * 0.1
    return A + A.T


# G of the two kernels: the same integrals in another order of summation, up
# to 1e5 terms of magnitude below 10 per element in FP64: below 1e-11 of the
# largest element (the engine's own bound against the oracle is 1e-10)
@pytest.mark.parametrize("name,basis", [("o2", "6-31g"), ("spread6", "6-31g"), ("spread40", "6-31g"),
                                        ("oh", "6-31+g**"), ("alkane3", "sto-3g")])
@pytest.mark.parametrize("target", [0, 8, 96])
def test_grouped_build_matches_oracle(monkeypatch, name, basis, target):
    monkeypatch.setenv("HFG_GROUP_MIN_TASKS", "0")
    Z, xyz = MOLECULES[name]
    eng = E.Engine(Z, xyz, basis, schwarz_threshold=0.0)
    eng.set_prim_target(target)  # lane groups of 1, up to 32 and a few lanes
    mol = O.Molecule(Z, xyz, basis_path(basis))
    packed = O.eri_packed(mol)
    P = _density(eng.nbf, 3)
    want = O.g_rhf(eng.nbf, packed, P)
    assert np.abs(eng.fock_rhf(P) - want).max() < 1e-11 * max(1.0, np.abs(want).max())
    Pb = _density(eng.nbf, 4)
    for got, ref in zip(eng.fock_uhf(P, Pb), O.g_uhf(eng.nbf, packed, P, Pb)):
        assert np.abs(got - ref).max() < 1e-11 * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("waters,basis", [(2, "6-31g*"), (5, "6-31g*"), (9, "6-31g")])
def test_grouped_build_matches_one_bra_per_task(monkeypatch, waters, basis):
    Z, xyz = molecules.water_cluster(waters, seed=waters)
    plain = E.Engine(Z, xyz, basis)
    monkeypatch.setenv("HFG_GROUP_MIN_TASKS", "0")
    grouped = E.Engine(Z, xyz, basis)
    assert plain.stats()["shell_quartets"] == grouped.stats()["shell_quartets"]
    P = _density(plain.nbf, 1)
    want = plain.fock_rhf(P)
    tol = 1e-11 * max(1.0, np.abs(want).max())
    assert np.abs(grouped.fock_rhf(P) - want).max() < tol
    grouped.set_streams(True)
    assert np.abs(grouped.fock_rhf(P) - want).max() < tol
    total = np.zeros_like(want)
    for rank in range(3):
        grouped.set_shard(rank, 3)
        total += grouped.fock_rhf(P)
    assert np.abs(total - want).max() < tol


def test_grouped_batch_with_inactive_molecules(monkeypatch):
    import torch
    mols = [(*molecules.water_cluster(k, seed=k), "6-31g") for k in (1, 3, 2)] + [(*molecules.alkane(2), "sto-3g")]
    plain = E.BatchEngine(mols)
    monkeypatch.setenv("HFG_GROUP_MIN_TASKS", "0")
    grouped = E.BatchEngine(mols)
    P = torch.from_numpy(np.concatenate([_density(int(n), i).ravel() for i, n in enumerate(plain.nbf)])).cuda()
    for active in ([1, 1, 1, 1], [1, 0, 1, 0]):
        a = torch.tensor(active, dtype=torch.uint8, device="cuda")
        out = [torch.zeros(plain.total, dtype=torch.float64, device="cuda") for _ in range(3)]
        plain.fock_rhf(P, out[0], active=active)
        grouped.fock_rhf(P, out[1], active=active)
        grouped.fock_rhf_async(P, out[2], a)
        torch.cuda.synchronize()
        for g in out[1:]:
            assert (g - out[0]).abs().max().item() < 1e-11 * max(1.0, out[0].abs().max().item())
