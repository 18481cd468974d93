"""The per-step engine with each panel beside the update before it (from 400
sites), at ragged last blocks and for the requests that change the matrix's
shape, against the oracle and against the same steps in turn (a call with kernel
timing takes them in turn).  Tolerance 1e-11 on S, the bound of every FP64 result
of this library; both orders do the same arithmetic on every element."""
import numpy as np
import pytest

import rgf_b200
from oracle.rgf_ref import cal_smatrix_RGF
from rgf_b200 import _abi

pytestmark = pytest.mark.gpu

TOL_S = 1e-11
FULL = ["left", "right"]


@pytest.mark.parametrize("in_", [FULL, ["left"]], ids=["full", "from_left"])
@pytest.mark.parametrize("ny", [399, 400, 401, 416, 447, 449, 600])
def test_matches_oracle_and_steps_in_turn(ny, in_):
    rng = np.random.default_rng(ny)
    s = dict(epsilon=1.0 + 3.0 * rng.random((ny, 4)), epsilon_L=1.0, epsilon_R=2.25, k0dx=2 * np.pi / 17,
             yBC="periodic" if ny % 2 else "Dirichlet")
    h = _abi.Handle(0)
    S, _ = rgf_b200.cal_smatrix_RGF(s, FULL, in_, options=_abi.Options(_abi.RGF_FP64, 1, 0, 0), handle=h)
    assert h.engine()[0] == 1 and h.stats()[1] < 1e-10
    S1, _ = rgf_b200.cal_smatrix_RGF(s, FULL, in_, options=_abi.Options(_abi.RGF_FP64, 1, 0, 1), handle=h)
    S0, _ = cal_smatrix_RGF(s, FULL, in_)
    assert np.linalg.norm(S - S0) <= TOL_S * np.linalg.norm(S0)
    assert np.linalg.norm(S - S1) <= TOL_S * np.linalg.norm(S0)
