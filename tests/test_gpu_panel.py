"""The per-step engine's cluster panel (whole-column pivoting in the registers
of one thread-block cluster), at the sizes where it changes shape.

Active rows per step are N plus the output channels carried; 64 rows a CTA is
the aim, so the cluster grows from 1 to 16 CTAs between 64 and 1024 active
rows, the CTA to 128 rows (512 threads) at 2048 and to 256 rows at 4096, and
wider matrices take the one-CTA panel in global memory.  Tolerance 1e-11 on S,
the bound of every FP64 result of this library against the oracle; measured
errors grow like sqrt(N) eps and stay below 1e-13.
"""
import numpy as np
import pytest

import rgf_b200
from oracle.rgf_ref import cal_smatrix_RGF as oracle

pytestmark = pytest.mark.gpu

TOL_S = 1e-11


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def structure(ny, nx, bc="Dirichlet", seed=0, eps_R=1.0, lam=15.0):
    rng = np.random.default_rng([seed, ny])
    return dict(epsilon=1.0 + 3.0 * rng.random((ny, nx)), epsilon_L=1.0, epsilon_R=eps_R, k0dx=2 * np.pi / lam, yBC=bc)


# (one channel carried per side of 'transmission': active rows are ny + few)
@pytest.mark.parametrize("ny", [1, 2, 31, 32, 33, 55, 63, 64, 65, 113, 128, 129, 225, 256, 257, 449, 511, 513, 900, 1025])
@pytest.mark.parametrize("form", ["full", "transmission"])
def test_cluster_panel_sizes(ny, form):
    s = structure(ny, 2, "periodic" if form == "full" else "Neumann", eps_R=1.0 if form == "full" else 2.25)
    out, in_ = (["left", "right"], ["left", "right"]) if form == "full" else (["right"], ["left"])
    S0, _ = oracle(s, out, in_)
    S, _ = rgf_b200.cal_smatrix_RGF(s, out, in_, options={"engine": 1})
    assert S.shape == S0.shape and S.size
    assert rel(S, S0) <= TOL_S


@pytest.mark.parametrize("ny", [1800, 2056])
def test_cluster_panel_wide(ny):
    """128 and 256 rows a CTA; a wide wavelength keeps the oracle's channel blocks small."""
    s = structure(ny, 1, lam=200.0)
    S0, _ = oracle(s, ["left", "right"], ["left"])
    S, _ = rgf_b200.cal_smatrix_RGF(s, ["left", "right"], ["left"])
    assert rel(S, S0) <= TOL_S


def test_panel_beyond_the_cluster():
    """Wider than 4096 active rows: a homogeneous slab transmits every channel
    with exp(i kx (nx + 1)) and reflects nothing."""
    ny, nx = 4100, 1
    s = dict(epsilon=np.ones((ny, nx)), epsilon_L=1.0, epsilon_R=1.0, k0dx=2 * np.pi / 400, yBC="Dirichlet")
    S, ch = rgf_b200.cal_smatrix_RGF(s, ["left", "right"], ["left"])
    kx = ch["L"]["kxdx"][ch["L"]["ind_prop"] - 1]
    n = len(kx)
    want = np.concatenate([np.zeros((n, n)), np.diag(np.exp(1j * kx * (nx + 1)))])
    assert np.abs(S - want).max() <= TOL_S


@pytest.mark.parametrize("ny", [1, 5, 32, 40, 64, 66, 100, 200, 300, 515, 1060])
def test_exchanges_across_the_cluster(ny):
    """Random segment states make the interface matrix P = I - g_R g_L a dense
    random one, whose pivots come from anywhere in the column.  The merged
    corner is Y + Z P^-1 X in numpy; a backward-stable elimination of order n
    is off by at most about n eps cond(P) of |Z P^-1 X|."""
    from rgf_b200.segments import DeviceSegments
    rng = np.random.default_rng(ny)
    s = structure(ny, 2)
    seg = DeviceSegments(s, ["left", "right"], ["left", "right"])
    (noL, niL), (noR, niR) = seg._sides

    def state(no, ni):
        return rng.standard_normal((ny + no, ny + ni)) + 1j * rng.standard_normal((ny + no, ny + ni))

    sL, sR = state(noL, niL), state(noR, niR)
    gL, XL, ZL, YL = sL[:ny, :ny], sL[:ny, ny:], sL[ny:, :ny], sL[ny:, ny:]
    gR, XR, ZR, YR = sR[:ny, :ny], sR[:ny, ny:], sR[ny:, :ny], sR[ny:, ny:]
    P = np.eye(ny) - gR @ gL
    X = np.concatenate([gR @ XL, XR], 1)
    Z = np.concatenate([ZL, ZR @ gL], 0)
    Y = np.block([[YL, np.zeros((noL, niR))], [ZR @ XL, YR]])
    V = np.linalg.solve(P, X)
    want = -2j * (Y + Z @ V)
    want[:noL, :niL] -= np.eye(noL, niL)
    want[noL:, niL:] -= np.eye(noR, niR)
    S = seg.merge(sL, sR)
    bound = 2 * np.finfo(float).eps * ny * np.linalg.cond(P) * np.linalg.norm(Z) * np.linalg.norm(V)
    assert np.linalg.norm(S - want) <= 10 * bound + 1e-13 * np.linalg.norm(want)
