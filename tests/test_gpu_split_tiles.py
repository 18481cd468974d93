"""The split-precision form's Gauss-Jordan step with two 128-column halves per
CTA (wide slices, from about 1000 sites) at a half that is empty, ragged and
full, against the FP64 form of the same structure.  Tolerance 1e-10 on S, the
bound of the split form; the refinement's own result has to stand."""
import numpy as np
import pytest

import rgf_b200
from rgf_b200 import _abi

pytestmark = pytest.mark.gpu

TOL_S = 1e-10


@pytest.mark.parametrize("ny", [980, 1024, 1030, 1088, 1100])
def test_wide_slices_match_fp64(ny):
    rng = np.random.default_rng(ny)
    s = dict(epsilon=1.0 + 2.0 * rng.random((ny, 9)), epsilon_L=1.0, epsilon_R=2.25, k0dx=2 * np.pi / 20,
             yBC="periodic")
    h = _abi.Handle(0)
    S, _ = rgf_b200.cal_smatrix_RGF(s, ["left", "right"], ["left"], options={"precision": _abi.RGF_TF32X3}, handle=h)
    assert h.refinement()["form"] == _abi.RGF_TF32X3
    S0, _ = rgf_b200.cal_smatrix_RGF(s, ["left", "right"], ["left"], handle=h)
    assert np.linalg.norm(S - S0) <= TOL_S * np.linalg.norm(S0)
