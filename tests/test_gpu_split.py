"""A structure swept in parts side by side (engine 0, S-matrices): the parts
and joins at the sizes where their number, tiles or shapes change, against the
oracle.  Tolerance 1e-11 on S, the bound of every FP64 result of this library;
joining adds one N-pivot elimination per part to the L of the sweep, so the
measured errors stay those of the unsplit sweep (1e-15 to 1e-13)."""
import numpy as np
import pytest

import rgf_b200
from oracle.rgf_ref import cal_smatrix_RGF, cal_smatrix_RGF_3D
from rgf_b200 import _abi

pytestmark = pytest.mark.gpu

TOL_S = 1e-11
FULL = ["left", "right"]
REQUESTS = {"full": (FULL, FULL), "from_left": (FULL, ["left"]), "transmission": (["right"], ["left"]),
            "back": (["left"], ["right"]), "reflection": (["left"], ["left"])}


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def structure(ny, nx, bc="periodic", eps_R=1.0, eta=0.0, lossy=False):
    rng = np.random.default_rng([ny, nx])
    eps = 1.0 + 3.0 * rng.random((ny, nx))
    if lossy:
        eps = eps + 0.02j * rng.random((ny, nx))
    return dict(epsilon=eps, epsilon_L=1.0, epsilon_R=eps_R, k0dx=2 * np.pi / 15 * (1 + 1j * eta if eta else 1), yBC=bc)


def unsplit(s, out, in_):
    """The same call in one sweep (a call that asks for kernel timing is never split)."""
    return rgf_b200.cal_smatrix_RGF(s, out, in_, options=_abi.Options(_abi.RGF_FP64, 0, 0, 1))[0]


@pytest.mark.parametrize("nx", [1, 3, 4, 5, 7, 33, 64])
@pytest.mark.parametrize("ny", [1, 2, 16, 31, 32, 33, 64, 65, 97, 150])
def test_parts_match_oracle(ny, nx):
    bc = {0: "periodic", 1: "Neumann", 2: "DirichletNeumann"}[nx % 3]
    s = structure(ny, nx, bc, eps_R=2.25 if nx % 2 else 1.0, eta=1e-3 if nx == 33 else 0.0, lossy=nx == 7)
    h = _abi.Handle(0)
    S, _ = rgf_b200.cal_smatrix_RGF(s, FULL, FULL, handle=h)
    S0, _ = cal_smatrix_RGF(s, FULL, FULL)
    assert rel(S, S0) <= TOL_S
    assert rel(S, unsplit(s, FULL, FULL)) <= TOL_S
    assert h.engine()[:2] == (0, 0) and h.stats()[1] < 1e-10


@pytest.mark.parametrize("form", sorted(REQUESTS))
@pytest.mark.parametrize("ny,nx", [(40, 50), (70, 21), (260, 12), (520, 8)])
def test_requests_match_oracle(ny, nx, form):
    out, in_ = REQUESTS[form]
    s = structure(ny, nx, "Dirichlet", eps_R=1.5)
    S, _ = rgf_b200.cal_smatrix_RGF(s, out, in_)
    S0, _ = cal_smatrix_RGF(s, out, in_)
    assert S.shape == S0.shape and rel(S, S0) <= TOL_S


def test_repeated_and_unequal_channel_lists():
    s = structure(48, 40, eps_R=2.0)
    out = {"ind_out_L": [3, 1, 3], "ind_out_R": [2]}
    in_ = {"ind_in_L": [1], "ind_in_R": [5, 4, 3, 3, 2, 1, 1]}
    S, _ = rgf_b200.cal_smatrix_RGF(s, out, in_)
    S0, _ = cal_smatrix_RGF(s, out, in_)
    assert rel(S, S0) <= TOL_S


@pytest.mark.parametrize("shape", [(3, 5, 30), (9, 8, 24), (17, 16, 9)])
def test_parts_in_3d(shape):
    rng = np.random.default_rng(shape)
    s = dict(epsilon=np.where(rng.random(shape) < 0.4, 2.25, 1.0), epsilon_L=1.0, epsilon_R=1.3, k0dx=2 * np.pi / 9,
             xyBC=[0.3, 0.7])
    S, _ = rgf_b200.cal_smatrix_RGF_3D(s, FULL, FULL)
    S0, _ = cal_smatrix_RGF_3D(s, FULL, FULL)
    assert rel(S, S0) <= TOL_S


def test_unitary_and_reciprocal_in_many_parts():
    """Real permittivity, many parts: S is unitary and symmetric under ind_prop_conj."""
    s = structure(60, 400)
    S, ch = rgf_b200.cal_smatrix_RGF(s, FULL, FULL)
    assert np.linalg.norm(S.conj().T @ S - np.eye(len(S))) <= 1e-11
    n = ch["L"]["N_prop"]
    p = np.concatenate([ch["L"]["ind_prop_conj"] - 1, n + ch["R"]["ind_prop_conj"] - 1])
    assert np.linalg.norm(S[p] - S[p].T) <= 1e-11


def test_a_part_that_fails_its_check_is_swept_whole():
    """Slice matrices that are singular behind a lead but not behind the slices
    before them: only an inner part meets one, its check fails, and the call is
    swept as one."""
    from tests.test_gpu_pivot import singular_slice_eps
    k0dx = 2 * np.pi / 15
    bad = singular_slice_eps(64, 2, k0dx)[:, :1]
    eps = np.repeat(bad, 200, axis=1)
    rng = np.random.default_rng(1)
    for k in (0, 1, -2, -1):
        eps[:, k] = 1 + 2 * rng.random(64)
    s = dict(epsilon=eps, epsilon_L=1.0, epsilon_R=1.0, k0dx=k0dx, yBC="Dirichlet")
    h = _abi.Handle(0)
    S, _ = rgf_b200.cal_smatrix_RGF(s, FULL, FULL, handle=h)
    S0, _ = cal_smatrix_RGF(s, FULL, FULL)
    assert rel(S, S0) <= TOL_S
    assert h.engine()[:2] == (0, 0) and h.stats()[1] < 1e-10


def test_nonfinite_permittivity_is_refused():
    s = structure(64, 100)
    s["epsilon"][5, 50] = np.nan
    with pytest.raises(Exception, match="NaN or Inf"):
        rgf_b200.cal_smatrix_RGF(s, FULL, FULL)


@pytest.mark.parametrize("checkpoint", [0, 1, 2, 7, 100])
@pytest.mark.parametrize("ny,nx", [(1, 4), (20, 5), (33, 31), (70, 12), (130, 9)])
def test_gradient_of_two_halves(ny, nx, checkpoint):
    """Odd cuts, short last segments, several segments side by side, and (at
    ny = 130, full S) the separate contraction for many channels; 1e-10 on the
    gradient, as for the one-sweep form."""
    from oracle.adjoint import grad_rgf_2d
    form = ("full", "transmission", "back", "from_left", "full")[[1, 20, 33, 70, 130].index(ny)]
    out, in_ = REQUESTS[form]
    s = structure(ny, nx, "periodic" if ny != 33 else "Neumann", eps_R=1.0 if ny == 130 else 2.0, lossy=nx == 31)
    rng = np.random.default_rng(ny)
    shape = cal_smatrix_RGF(s, out, in_)[0].shape
    D = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    S0, g0 = grad_rgf_2d(s, out, in_, D)
    S, g = rgf_b200.smatrix_grad_RGF(s, out, in_, D, checkpoint=checkpoint)
    assert rel(S, S0) <= TOL_S
    assert np.abs(g - g0).max() <= 1e-10 * np.abs(g0).max()


@pytest.mark.parametrize("form", sorted(REQUESTS))
@pytest.mark.parametrize("ny,nx", [(20, 4), (34, 11)])
def test_fields_of_two_halves(ny, nx, form):
    from oracle.dense_fdfd import fields_dense_2d
    out, in_ = REQUESTS[form]
    s = structure(ny, nx, 0.4, eps_R=1.7)
    _, psi0 = fields_dense_2d(s, out, in_)
    for checkpoint in (0, 3):
        S, psi = rgf_b200.fields_RGF(s, out, in_, checkpoint=checkpoint)
        assert np.linalg.norm(psi - psi0) <= TOL_S * np.linalg.norm(psi0)


def test_gradient_on_the_device_in_two_halves():
    """S, weights, gradient and fields as device buffers, one handle for calls of changing size."""
    import ctypes

    import torch
    from rgf_b200.api import _request
    h = _abi.Handle(0)
    for ny, nx in ((48, 21), (16, 40), (90, 8)):
        s = structure(ny, nx)
        req, keep = _request(FULL, FULL)
        S0, _ = cal_smatrix_RGF(s, FULL, FULL)
        n = S0.shape[0]
        eps = torch.from_numpy(np.ascontiguousarray(np.asarray(s["epsilon"], complex).ravel(order="F"))).cuda()
        sy = _abi.Syst2D(ny, nx, eps.data_ptr(), 1, _abi.cplx(1.0), _abi.cplx(1.0), _abi.cplx(s["k0dx"]),
                         _abi.BC_PERIODIC, 0.0)
        D = torch.from_numpy(np.ascontiguousarray(np.conj(S0).T)).cuda()
        S = torch.zeros((n, n), dtype=torch.complex128, device="cuda")
        g = torch.zeros((nx, ny), dtype=torch.complex128, device="cuda")
        opt = _abi.Options(_abi.RGF_FP64, 0, 1, 0)
        torch.cuda.synchronize()
        _abi.check(h.lib.rgf_smatrix_grad_2d(h.h, ctypes.byref(sy), ctypes.byref(req), ctypes.byref(opt), D.data_ptr(), n,
                                             S.data_ptr(), n, g.data_ptr(), 4))
        host = rgf_b200.smatrix_grad_RGF(s, FULL, FULL, np.conj(S0), checkpoint=4)
        assert rel(S.cpu().numpy().T, S0) <= TOL_S
        assert rel(g.cpu().numpy().T, host[1]) <= 1e-12
        del keep
