"""Shards of one build whose ranks differ in settings that choose kernels, not
results (class streams, per-class timing): the partial G still sum to the full
one.  The task limit is set so that the largest classes lie between the two
lines of the grouped kernel (as it is, and twice that on class streams), where
a context's builds run either kernel of a class."""
import numpy as np
import pytest
import torch

from hartreefock_b200 import engine as E
from hartreefock_b200 import molecules

pytestmark = pytest.mark.gpu

BASIS = "6-31g*"


def _density(n, seed):
    A = np.random.default_rng(seed).normal(size=(n, n)) * 0.1
    return A + A.T


def _limit(Z, xyz):
    """Tasks per SM that two thirds of the largest fused class's tasks come to."""
    eng = E.Engine(Z, xyz, BASIS)
    eng.set_profiling(True)
    eng.fock_rhf(np.eye(eng.nbf))
    most = max(c["tasks"] for c in eng.class_profile() if c["la"] + c["lb"] + c["lc"] + c["ld"] <= 2)
    return str(max(1, 2 * most // (3 * torch.cuda.get_device_properties(0).multi_processor_count)))


def _settings(Z, xyz):
    """Engines of the same molecule and options: defaults, class streams, timing, both."""
    out = []
    for streams, timing in ((False, False), (True, False), (False, True), (True, True)):
        eng = E.Engine(Z, xyz, BASIS)
        eng.set_streams(streams)
        eng.set_profiling(timing)
        out.append(eng)
    return out


# the same integrals in another order of summation: below 1e-11 of the largest
# element of G, as for shards with equal settings
@pytest.mark.parametrize("waters", [5, 9])
def test_shards_with_different_settings_sum_to_the_full_build(monkeypatch, waters):
    Z, xyz = molecules.water_cluster(waters, seed=2)
    monkeypatch.setenv("HFG_GROUP_MIN_TASKS", "1000000000")
    plain = E.Engine(Z, xyz, BASIS)
    P, Pb = _density(plain.nbf, 1), _density(plain.nbf, 2)
    full = plain.fock_rhf(P)
    fa, fb = plain.fock_uhf(P, Pb)
    monkeypatch.setenv("HFG_GROUP_MIN_TASKS", _limit(Z, xyz))
    engines = _settings(Z, xyz)
    for eng in engines:  # either kernel gives the unsharded build
        assert np.abs(eng.fock_rhf(P) - full).max() < 1e-11 * max(1.0, np.abs(full).max())
    for count in (2, 4):
        total, ga, gb = np.zeros_like(full), np.zeros_like(full), np.zeros_like(full)
        for r in range(count):
            eng = engines[r]
            eng.set_shard(r, count)
            total += eng.fock_rhf(P)
            a, b = eng.fock_uhf(P, Pb)
            ga += a
            gb += b
        assert np.abs(total - full).max() < 1e-11 * max(1.0, np.abs(full).max())
        for got, want in ((ga, fa), (gb, fb)):
            assert np.abs(got - want).max() < 1e-11 * max(1.0, np.abs(want).max())


def test_one_context_switched_between_its_shards(monkeypatch):
    Z, xyz = molecules.water_cluster(6, seed=4)
    monkeypatch.setenv("HFG_GROUP_MIN_TASKS", _limit(Z, xyz))
    eng = E.Engine(Z, xyz, BASIS)
    P = _density(eng.nbf, 3)
    full = eng.fock_rhf(P)
    total = np.zeros_like(full)
    for r in range(2):
        eng.set_shard(r, 2)
        eng.set_streams(r == 1)
        total += eng.fock_rhf(P)
    assert np.abs(total - full).max() < 1e-11 * max(1.0, np.abs(full).max())
