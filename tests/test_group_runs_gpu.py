"""The grouped class kernels with runs of 1, 3 and 16 bras per task, whatever
the molecule's size: against the oracle and the one-bra-per-task kernels, RHF
and UHF, with d shells, in shards and in batches.  The class profile says that
they ran."""
import numpy as np
import pytest

import oracle as O
from hartreefock_b200 import engine as E
from hartreefock_b200 import molecules
from hartreefock_b200.basis_io import basis_path

pytestmark = pytest.mark.gpu

GROUPED = {(0, 0, 0, 0), (1, 0, 0, 0), (1, 0, 1, 0), (1, 1, 0, 0), (1, 1, 1, 0), (2, 0, 0, 0), (2, 0, 1, 0), (2, 1, 0, 0)}
O2 = ([8, 8], np.array([[0.0, 0.0, 0.0], [0.3, -0.2, 2.3]]))


def _density(n, seed):
    A = np.random.default_rng(seed).normal(size=(n, n)) * 0.1
    return A + A.T


def _plain(monkeypatch, make):
    monkeypatch.setenv("HFG_GROUP_MIN_TASKS", "1000000000")
    return make()


def _grouped(monkeypatch, make, run):
    monkeypatch.setenv("HFG_GROUP_MIN_TASKS", "0")
    monkeypatch.setenv("HFG_GROUP_RUN", str(run))
    return make()


def _kernels(eng):
    """(grouped classes, all classes that have the kernel) of the engine's builds."""
    prof = eng.class_profile()
    have = {(c["la"], c["lb"], c["lc"], c["ld"]) for c in prof} & GROUPED
    return {(c["la"], c["lb"], c["lc"], c["ld"]) for c in prof if c["grouped"]}, have


# the engine's bound against the oracle: 1e-10 of the largest element of G
@pytest.mark.parametrize("run", [1, 3, 16])
@pytest.mark.parametrize("mol,basis", [(O2, "6-31g*"), (molecules.hydroxyl(), "6-31+g**"),
                                       (molecules.water_cluster(1, seed=3), "6-31g*")])
def test_runs_match_the_oracle(monkeypatch, mol, basis, run):
    eng = _grouped(monkeypatch, lambda: E.Engine(*mol, basis, schwarz_threshold=0.0), run)
    used, have = _kernels(eng)
    assert used == have == GROUPED
    packed = O.eri_packed(O.Molecule(*mol, basis_path(basis)))
    P, Pb = _density(eng.nbf, 3), _density(eng.nbf, 4)
    want = O.g_rhf(eng.nbf, packed, P)
    assert np.abs(eng.fock_rhf(P) - want).max() < 1e-10 * max(1.0, np.abs(want).max())
    for got, ref in zip(eng.fock_uhf(P, Pb), O.g_uhf(eng.nbf, packed, P, Pb)):
        assert np.abs(got - ref).max() < 1e-10 * max(1.0, np.abs(ref).max())


# two kernels of the same quartets in FP64, up to 1e5 terms of magnitude below
# 10 per element in another order: 1e-11 of the largest element.  The chain's
# ends do not overlap: runs hold bras that reach none of a task's kets.
@pytest.mark.parametrize("run", [1, 3, 16])
@pytest.mark.parametrize("mol,basis", [(molecules.alkane(8), "6-31g*"), (molecules.alkane(4), "6-31+g**"),
                                       (molecules.water_cluster(5, seed=1), "6-31g*")])
def test_runs_match_one_bra_per_task(monkeypatch, mol, basis, run):
    plain = _plain(monkeypatch, lambda: E.Engine(*mol, basis))
    assert not _kernels(plain)[0]
    P, Pb = _density(plain.nbf, 1), _density(plain.nbf, 2)
    want = [plain.fock_rhf(P), *plain.fock_uhf(P, Pb)]
    eng = _grouped(monkeypatch, lambda: E.Engine(*mol, basis), run)
    used, have = _kernels(eng)
    assert used == have
    total = [np.zeros_like(w) for w in want]
    for count in (1, 3):
        total = [np.zeros_like(w) for w in want]
        for r in range(count):
            eng.set_shard(r, count)
            for t, g in zip(total, [eng.fock_rhf(P), *eng.fock_uhf(P, Pb)]):
                t += g
        for t, w in zip(total, want):
            assert np.abs(t - w).max() < 1e-11 * max(1.0, np.abs(w).max())


@pytest.mark.parametrize("run", [3, 16])
def test_runs_in_a_batch(monkeypatch, run):
    import torch
    mols = [(*molecules.water_cluster(k, seed=k), "6-31g*") for k in (1, 3, 2)] + [(*molecules.alkane(2), "6-31+g**")]
    plain = _plain(monkeypatch, lambda: E.BatchEngine(mols))
    grouped = _grouped(monkeypatch, lambda: E.BatchEngine(mols), run)
    Pa, Pb = (torch.from_numpy(np.concatenate([_density(int(n), i + s).ravel() for i, n in enumerate(plain.nbf)])).cuda()
              for s in (0, 10))
    for active in ([1, 1, 1, 1], [0, 1, 0, 1]):
        a = torch.tensor(active, dtype=torch.uint8, device="cuda")
        new = lambda: torch.zeros(plain.total, dtype=torch.float64, device="cuda")
        want, wa, wb = new(), new(), new()
        plain.fock_rhf(Pa, want, active=active)
        plain.fock_uhf(Pa, Pb, wa, wb, active=active)
        for asynchronous in (False, True):
            g, ga, gb = new(), new(), new()
            if asynchronous:
                grouped.fock_rhf_async(Pa, g, a)
                grouped.fock_uhf_async(Pa, Pb, ga, gb, a)
            else:
                grouped.fock_rhf(Pa, g, active=active)
                grouped.fock_uhf(Pa, Pb, ga, gb, active=active)
            torch.cuda.synchronize()
            for got, ref in ((g, want), (ga, wa), (gb, wb)):
                assert (got - ref).abs().max().item() < 1e-11 * max(1.0, ref.abs().max().item())
