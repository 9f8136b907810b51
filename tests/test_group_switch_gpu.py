"""A context that turns from the precision form to plain builds runs the same
kernels, and cuts the same shards, as one that was plain from the start."""
import numpy as np
import pytest

from hartreefock_b200 import engine as E
from hartreefock_b200 import molecules

pytestmark = pytest.mark.gpu


# the same integrals in another order of summation: 1e-11 of the largest element
@pytest.mark.parametrize("graphs", [False, True])
@pytest.mark.parametrize("form", [{"incremental": True}, {"mixed_cutoff": 1e-4}])
def test_plain_builds_after_the_precision_form(monkeypatch, form, graphs):
    Z, xyz = molecules.water_cluster(4, seed=6)
    monkeypatch.setenv("HFG_GROUP_MIN_TASKS", "0")
    monkeypatch.setenv("HFG_GROUP_RUN", "3")
    plain = E.Engine(Z, xyz, "6-31g*")
    A = np.random.default_rng(1).normal(size=(plain.nbf, plain.nbf)) * 0.1
    P = A + A.T
    want = plain.fock_rhf(P)
    tol = 1e-11 * max(1.0, np.abs(want).max())
    eng = E.Engine(Z, xyz, "6-31g*", **form)
    eng.set_graphs(graphs)
    eng.fock_rhf(P)
    assert not any(c["grouped"] for c in eng.class_profile())
    eng.set_incremental(False)
    eng.set_mixed_cutoff(0.0)
    for _ in range(3):
        assert np.abs(eng.fock_rhf(P) - want).max() < tol
    assert {k: c["grouped"] for k, c in enumerate(eng.class_profile())} == \
           {k: c["grouped"] for k, c in enumerate(plain.class_profile())}
    plain.set_shard(0, 2)
    eng.set_shard(1, 2)
    assert np.abs(plain.fock_rhf(P) + eng.fock_rhf(P) - want).max() < tol
