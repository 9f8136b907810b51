"""The large classes' kernel by primitive quartets: builds on either side of the
lines agree with the split path."""
import numpy as np
import pytest

from hartreefock_b200 import engine as E
from hartreefock_b200 import molecules

pytestmark = pytest.mark.gpu


# two evaluations of the same integrals in FP64: below 1e-11 of the largest
# element of G (the engine's bound against the oracle is 1e-10)
@pytest.mark.parametrize("waters", [1, 3, 6, 9])
def test_default_kernels_match_the_split_path(monkeypatch, waters):
    Z, xyz = molecules.water_cluster(waters, seed=waters)
    auto = E.Engine(Z, xyz, "6-31g*", eri_convention=E.ERI_EXACT)
    monkeypatch.setenv("HFG_SPLIT_PATH", "1")
    split = E.Engine(Z, xyz, "6-31g*", eri_convention=E.ERI_EXACT)
    A = np.random.default_rng(waters).normal(size=(auto.nbf, auto.nbf)) * 0.1
    P = A + A.T
    want = split.fock_rhf(P)
    assert np.abs(auto.fock_rhf(P) - want).max() < 1e-11 * max(1.0, np.abs(want).max())
    for got, ref in zip(auto.fock_uhf(P, 0.5 * P), split.fock_uhf(P, 0.5 * P)):
        assert np.abs(got - ref).max() < 1e-11 * max(1.0, np.abs(ref).max())
