"""Which kernel a large class runs by default, on either side of the lines, as
the class profile reports it."""
import numpy as np
import pytest

from hartreefock_b200 import engine as E
from hartreefock_b200 import molecules

pytestmark = pytest.mark.gpu


def _on_warp(mol, basis):
    eng = E.Engine(*mol, basis, eri_convention=E.ERI_EXACT)
    eng.set_profiling(True)
    eng.fock_rhf(np.eye(eng.nbf))
    return {(c["la"], c["lb"], c["lc"], c["ld"]) for c in eng.class_profile() if c["warp_kernel"]}


# (dp|ds) and (dp|dp) keep the split path at every size; the others with few
# primitive quartets run the warp kernel
@pytest.mark.parametrize("mol,basis", [(molecules.water_cluster(1, seed=0), "6-31g*"),
                                       (molecules.water_cluster(2, seed=0), "6-31g*"),
                                       (molecules.methyl_planar(), "6-31+g**")])
def test_small_molecules(mol, basis):
    assert _on_warp(mol, basis) == {(2, 2, 2, 2), (2, 2, 2, 1), (2, 2, 2, 0), (2, 2, 1, 1), (2, 2, 1, 0),
                                    (2, 1, 1, 1)}


def test_above_every_line():
    assert _on_warp(molecules.water_cluster(18, seed=0), "6-31g*") == {(2, 2, 2, 2)}
