"""Channel set-up at the sizes where it changes form: one launch with a CTA per
side up to 8192 channels, one thread of the GPU per channel beyond; one and two
sides, equal and unlike leads.  The wave numbers are the same functions of the
same arguments in both, so the oracle's tolerance is that of the other channel
tests (1e-12 relative), and channel lists agree exactly."""
import numpy as np
import pytest

import rgf_b200
from oracle.rgf_ref import setup_channels, setup_channels_3D

pytestmark = pytest.mark.gpu


def same(a, b, key):
    assert a["N_prop"] == b["N_prop"]
    assert np.array_equal(a["ind_prop"], b["ind_prop"])
    if "ind_prop_conj" in b:
        assert np.array_equal(a["ind_prop_conj"], b["ind_prop_conj"])
    for k in (key, "sqrt_mu"):
        np.testing.assert_allclose(a[k], b[k], rtol=1e-12, atol=1e-13)


@pytest.mark.parametrize("ny", [1, 33, 1023, 1024, 1025, 8191, 8192, 8193, 20000])
@pytest.mark.parametrize("bc", ["periodic", "Neumann", 0.4])
def test_both_forms_2d(ny, bc):
    for eps_R in (None, 1.0, 2.25):
        k0dx = 2 * np.pi / 12 * (1 + 1e-3j if eps_R == 2.25 else 1)
        ours, ref = (f(ny, bc, k0dx, 1.0, eps_R) for f in (rgf_b200.setup_channels, setup_channels))
        np.testing.assert_allclose(ours["kydx"], ref["kydx"], rtol=1e-14, atol=1e-15)
        same(ours["L"], ref["L"], "kxdx")
        if eps_R is None:
            assert np.isnan(ours["R"]["N_prop"])
        else:
            same(ours["R"], ref["R"], "kxdx")


@pytest.mark.parametrize("shape", [(3, 5), (90, 91), (91, 91)])
def test_both_forms_3d(shape):
    ours, ref = (f(*shape, [0.3, 0.7], 2 * np.pi / 9, 1.0, 1.5) for f in (rgf_b200.setup_channels_3D, setup_channels_3D))
    np.testing.assert_allclose(ours["kydx"], ref["kydx"], rtol=1e-14, atol=1e-15)
    np.testing.assert_allclose(ours["kxdx"], ref["kxdx"], rtol=1e-14, atol=1e-15)
    for s in ("L", "R"):
        same(ours[s], ref[s], "kzdx")
