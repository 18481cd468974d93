"""The pivot-block inverses of the split-precision form at the widths where
their panels, padding and hand-over between slices change (blocks of 32, panels
of four columns, 128-row tiles), against the oracle.  Tolerance 1e-10 on S, the
bound of this form; the refinement's own result has to stand, which a wrong
pivot-block inverse does not allow (the factor would not contract)."""
import numpy as np
import pytest

import rgf_b200
from oracle.rgf_ref import cal_smatrix_RGF
from rgf_b200 import _abi

pytestmark = pytest.mark.gpu

TOL_S = 1e-10
FULL = ["left", "right"]


@pytest.mark.parametrize("nx", [2, 9])
@pytest.mark.parametrize("ny", [1, 3, 4, 5, 29, 31, 32, 33, 36, 63, 64, 65, 100, 127, 128, 129, 130])
def test_widths_match_oracle(ny, nx):
    rng = np.random.default_rng([ny, nx])
    s = dict(epsilon=1.0 + 3.0 * rng.random((ny, nx)), epsilon_L=1.0, epsilon_R=2.25, k0dx=2 * np.pi / 15,
             yBC="periodic" if nx == 2 else "Dirichlet")
    h = _abi.Handle(0)
    S, _ = rgf_b200.cal_smatrix_RGF(s, FULL, FULL, options={"precision": _abi.RGF_TF32X3}, handle=h)
    S0, _ = cal_smatrix_RGF(s, FULL, FULL)
    assert S.shape == S0.shape
    assert np.linalg.norm(S - S0) <= TOL_S * max(np.linalg.norm(S0), 1e-300)
    if S0.size:
        assert h.refinement()["form"] == _abi.RGF_TF32X3
