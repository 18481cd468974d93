"""The substitution sweeps of the split-precision form where their shape changes:
one and two sides (below and from 8 slices), the two tile widths and their edges
(32 and 64 columns), ragged K-splits, sites around a 128-row tile -- against the
oracle.  Tolerance 1e-10 on S, the bound of this form; the refinement's own
result has to stand, and in as few passes as a sweep of correct solves takes
(a wrong row, column or slice in a sweep would not contract)."""
import numpy as np
import pytest

import rgf_b200
from oracle.rgf_ref import cal_smatrix_RGF
from rgf_b200 import _abi

pytestmark = pytest.mark.gpu

TOL_S = 1e-10


@pytest.mark.parametrize("nx", [1, 7, 8])
@pytest.mark.parametrize("ny", [40, 128, 150])
@pytest.mark.parametrize("cols", [1, 32, 33, 64, 65, 130])
def test_sweeps_match_oracle(ny, nx, cols):
    rng = np.random.default_rng([ny, nx, cols])
    s = dict(epsilon=1.0 + 2.0 * rng.random((ny, nx)), epsilon_L=1.0, epsilon_R=2.25, k0dx=2 * np.pi / 12,
             yBC="Neumann" if nx == 8 else "periodic")
    in_ = {"ind_in_L": [1 + i % 6 for i in range(cols - cols // 3)], "ind_in_R": [1 + i % 6 for i in range(cols // 3)]}
    out = ["left", "right"]
    h = _abi.Handle(0)
    S, _ = rgf_b200.cal_smatrix_RGF(s, out, in_, options={"precision": _abi.RGF_TF32X3}, handle=h)
    S0, _ = cal_smatrix_RGF(s, out, in_)
    info = h.refinement()
    assert S.shape == S0.shape and np.linalg.norm(S - S0) <= TOL_S * np.linalg.norm(S0)
    assert info["form"] == _abi.RGF_TF32X3 and info["iterations"] <= 6
