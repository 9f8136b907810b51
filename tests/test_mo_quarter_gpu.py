"""The quarter transforms of the MO integrals against numpy, at orbital ranges
that need one and several slabs."""
import numpy as np
import pytest
import torch

import oracle as O
from hartreefock_b200 import engine as E
from hartreefock_b200 import molecules
from hartreefock_b200.basis_io import basis_path

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("i0,ni,a0,na", [(0, 1, 1, 1), (0, 5, 5, 8), (2, 3, 0, 13), (0, 13, 12, 1), (0, 13, 0, 13)])
def test_quarter_transforms_match_numpy(i0, ni, a0, na):
    Z, xyz = molecules.H2O_README
    eng = E.Engine(Z, xyz, "6-31g", schwarz_threshold=0.0)
    n = eng.nbf
    packed = O.eri_packed(O.Molecule(Z, xyz, basis_path("6-31g")))
    ij = np.array([[max(i, j) * (max(i, j) + 1) // 2 + min(i, j) for j in range(n)] for i in range(n)])
    hi, lo = np.maximum(ij[:, :, None, None], ij[None, None]), np.minimum(ij[:, :, None, None], ij[None, None])
    eri = packed[hi * (hi + 1) // 2 + lo]
    C = np.linalg.qr(np.random.default_rng(5).normal(size=(n, n)))[0]
    Ci, Ca = C[:, i0:i0 + ni], C[:, a0:a0 + na]
    want = np.einsum("mnls,mi,na,lj,sb->iajb", eri, Ci, Ca, Ci, Ca, optimize=True).reshape(ni * na, ni * na)
    X = eng.mo_eri_ovov_tensor(torch.from_numpy(C).cuda(), i0, ni, a0, na).cpu().numpy()
    again = eng.mo_eri_ovov_tensor(torch.from_numpy(C).cuda(), 0, 1, 0, 2).cpu().numpy()  # in the kept workspace
    small = np.einsum("mnls,mi,na,lj,sb->iajb", eri, C[:, :1], C[:, :2], C[:, :1], C[:, :2], optimize=True).reshape(2, 2)
    # 13^4 terms of magnitude below 5 with orthonormal coefficients, plus the
    # integrals' own 1e-12
    assert np.abs(X - want).max() < 2e-11
    assert np.abs(again - small).max() < 2e-11
