"""Densities with NaN or infinite entries: the grouped kernels leave the same
elements of G finite as the kernels with one bra per task, which touch an
element only through quartets of the build."""
import numpy as np
import pytest

from hartreefock_b200 import engine as E
from hartreefock_b200 import molecules

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("size,basis", [(12, "6-31g"), (8, "6-31g*")])
def test_nonfinite_entries_spread_no_further(monkeypatch, value, size, basis):
    Z, xyz = molecules.alkane(size)
    monkeypatch.setenv("HFG_GROUP_MIN_TASKS", "1000000000")
    plain = E.Engine(Z, xyz, basis)
    monkeypatch.setenv("HFG_GROUP_MIN_TASKS", "0")
    grouped = E.Engine(Z, xyz, basis)
    n = plain.nbf
    P = np.eye(n)
    P[n - 1, n - 1] = value
    want, got = plain.fock_rhf(P), grouped.fock_rhf(P)
    assert 0 < np.isfinite(want).sum() < want.size
    assert np.array_equal(np.isfinite(got), np.isfinite(want))
    wants, gots = plain.fock_uhf(np.eye(n), P), grouped.fock_uhf(np.eye(n), P)
    for g, w in zip(gots, wants):
        assert np.array_equal(np.isfinite(g), np.isfinite(w))
