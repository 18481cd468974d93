"""Cases for timing the public calls of rgf_b200.

A case is a dict of plain values.  ``kind`` says which call it makes:

  smatrix    cal_smatrix_RGF / cal_smatrix_RGF_3D
  grad       smatrix_grad_RGF
  fields     fields_RGF
  batch      cal_smatrix_RGF_batch
  channels   setup_channels

and the other entries give the structure: transverse size (``ny``, or ``nx`` x
``ny`` when ``dim`` is 3), ``slices``, boundary condition, permittivity,
leads, frequency, requested channels and precision form.  ``exact`` solves the
same discretised scattering problem in complex128 with torch, as one
block-tridiagonal system, without this repository's code.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import rgf_b200
from rgf_b200 import workloads

# permittivity distributions: i.i.d. uniform [1, 4) and [1, 3) (random media),
# two-phase voxels, disks in a background with absorption (disordered slabs),
# and uniform with absorption
EPSILONS = ("uniform4", "uniform3", "binary", "disks", "lossy")
BOUNDARIES = ("periodic", "Dirichlet", "Neumann", "DirichletNeumann", "NeumannDirichlet", "bloch")
REQUESTS = ("full", "from_left", "transmission", "first8")

_DEFAULTS = dict(kind="smatrix", dim=2, nx=1, bc="periodic", eps="uniform4", eps_L=1.0, eps_R=1.0,
                 pixels_per_wavelength=15.0, eta=0.0, request="full", precision=0, checkpoint=0, count=1)


def _case(**kw):
    return dict(_DEFAULTS, **kw)


def listed():
    return [
        # channel set-up of a wide waveguide on its own, as done before a request is chosen
        _case(name="channels_2d_501", kind="channels", ny=501, slices=0, eps_R=2.25),
        # the smallest S-matrix: a thin, short structure, one of many in a scan
        _case(name="small_2d_16x24", ny=16, slices=24, bc="Dirichlet"),
        # the ordinary small structure: 64 x 200 random medium, full S
        _case(name="plain_2d_64x200", ny=64, slices=200),
        # a transmission matrix between unlike leads, odd size, absorption
        _case(name="transmission_2d_157x263", ny=157, slices=263, bc="Neumann", eps="lossy", eps_R=2.25,
              request="transmission"),
        # one step of an inverse design: S and its gradient, 8 x 8 channels, a checkpoint every 23 slices
        _case(name="gradient_2d_256x512", kind="grad", ny=256, slices=512, request="first8", checkpoint=23),
        # the field of every incoming channel inside a slab
        _case(name="fields_2d_180x141", kind="fields", ny=180, slices=141, bc="bloch"),
        # a 3D photonic crystal slab, Bloch phases, both numeric forms
        _case(name="bloch_3d_24x24x300", dim=3, nx=24, ny=24, slices=300, bc="bloch", eps="binary",
              pixels_per_wavelength=12.0),
        _case(name="bloch_3d_24x24x300_tf32x3", dim=3, nx=24, ny=24, slices=300, bc="bloch", eps="binary",
              pixels_per_wavelength=12.0, precision=1),
        # the wide disordered waveguide, both numeric forms
        _case(name="disks_2d_1024x320", ny=1024, slices=320, bc="Dirichlet", eps="disks",
              pixels_per_wavelength=20.0),
        _case(name="disks_2d_1024x320_tf32x3", ny=1024, slices=320, bc="Dirichlet", eps="disks",
              pixels_per_wavelength=20.0, precision=1),
        # a waveguide wider than the widest one whose slice matrix stays on the chip
        _case(name="wide_2d_1500x20", ny=1500, slices=20, bc="Dirichlet", eps="disks",
              pixels_per_wavelength=20.0),
        # an ensemble of uneven structures at complex frequency, in one call
        _case(name="batch_2d_12", kind="batch", ny=512, slices=2000, eps="uniform3", eta=1e-3, count=12),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


_LARGEST = 3.5e12  # flops of one S-matrix of the largest listed cases


def draw(rng):
    kind = rng.choices(["smatrix2", "smatrix3", "tf32x3", "wide", "grad", "fields", "batch", "channels"],
                       [8, 2, 2, 1, 2, 2, 1, 1])[0]
    common = dict(pixels_per_wavelength=round(rng.uniform(10.0, 24.0), 2))
    if kind == "channels":
        return _case(kind="channels", ny=_log_int(rng, 20, 1500), slices=0, bc=rng.choice(BOUNDARIES),
                     eps_R=rng.choice([1.0, 2.25]), **common)
    if kind == "batch":
        return _case(kind="batch", ny=_log_int(rng, 100, 512), slices=_log_int(rng, 200, 1500), eps="uniform3",
                     eta=1e-3, count=rng.randint(2, 9), **common)
    if kind == "wide":
        return _case(ny=rng.randint(1100, 1700), slices=rng.randint(2, 20), bc="Dirichlet", eps="disks",
                     pixels_per_wavelength=20.0)
    if kind == "smatrix3":
        nx, ny = _log_int(rng, 3, 28), _log_int(rng, 3, 28)
        return _case(dim=3, nx=nx, ny=ny, slices=_log_int(rng, 10, 300), bc=rng.choice(["periodic", "Dirichlet", "bloch"]),
                     eps="binary", request=rng.choice(["full", "from_left"]), **common)
    if kind == "tf32x3":
        ny = _log_int(rng, 64, 1024)
        return _case(ny=ny, slices=_log_int(rng, 20, 320), bc="Dirichlet", eps="disks", pixels_per_wavelength=20.0,
                     precision=1)
    if kind == "grad":
        return _case(kind="grad", ny=_log_int(rng, 40, 400), slices=_log_int(rng, 20, 500), request="first8",
                     checkpoint=rng.choice([0, 0, 23]), bc=rng.choice(BOUNDARIES), eps=rng.choice(["uniform4", "lossy"]),
                     pixels_per_wavelength=15.0)
    if kind == "fields":
        return _case(kind="fields", ny=_log_int(rng, 32, 300), slices=_log_int(rng, 16, 200), bc=rng.choice(BOUNDARIES),
                     request=rng.choice(["full", "from_left"]), **common)
    ny = _log_int(rng, 8, 1050)
    slices = _log_int(rng, 8, 1500)
    while slices > 8 and 1.4 * slices * 8.0 * ny ** 3 > _LARGEST:
        slices //= 2
    return _case(ny=ny, slices=slices, bc=rng.choice(BOUNDARIES), eps=rng.choice(EPSILONS),
                 eps_R=rng.choice([1.0, 1.0, 2.25]), eta=rng.choice([0.0, 0.0, 5e-4]),
                 request=rng.choice(["full", "full", "from_left", "transmission"]), **common)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _permittivity(kind, shape, seed):
    rng = np.random.default_rng([7, seed])
    if kind == "uniform4":
        return 1.0 + 3.0 * rng.random(shape)
    if kind == "uniform3":
        return 1.0 + 2.0 * rng.random(shape)
    if kind == "binary":
        return np.where(rng.random(shape) < 0.4, 2.25, 1.0)
    if kind == "lossy":
        return 1.0 + 2.0 * rng.random(shape) + 0.01j * rng.random(shape)
    return workloads.disks_permittivity(shape[0], shape[1], seed)


def _boundary(case):
    if case["bc"] != "bloch":
        return case["bc"]
    return [0.3, 0.7] if case["dim"] == 3 else 0.4


def _k0dx(case):
    k = 2.0 * np.pi / case["pixels_per_wavelength"]
    return k * (1.0 + 1j * case["eta"]) if case["eta"] else k


def _request(case):
    return {"full": (["left", "right"], ["left", "right"]),
            "from_left": (["left", "right"], ["left"]),
            "transmission": (["right"], ["left"]),
            "first8": ({"ind_out_R": _first(case, 1)}, {"ind_in_L": _first(case, 0)})}[case["request"]]


def _first(case, side):
    """The first eight propagating channels of a lead (all, when it has fewer), 1-based."""
    return np.arange(1, min(8, len(_lead(case, side)["prop"])) + 1)


def _syst(case, seed):
    shape = (case["ny"], case["slices"]) if case["dim"] == 2 else (case["nx"], case["ny"], case["slices"])
    s = dict(epsilon=_permittivity(case["eps"], shape, seed), epsilon_L=case["eps_L"], epsilon_R=case["eps_R"],
             k0dx=_k0dx(case))
    s["yBC" if case["dim"] == 2 else "xyBC"] = _boundary(case)
    return s


def _batch_sizes(case):
    """Transverse size, slices and imaginary part of every structure: uneven,
    from a quarter (an eighth) of the largest size up."""
    rng = np.random.default_rng([11, case["ny"], case["slices"], case["count"]])
    ny = rng.integers(max(case["ny"] // 8, 2), case["ny"] + 1, size=case["count"])
    nx = rng.integers(max(case["slices"] // 20, 2), case["slices"] + 1, size=case["count"])
    eta = rng.uniform(0.0, case["eta"], size=case["count"])
    return [(int(a), int(b), float(c)) for a, b, c in zip(ny, nx, eta)]


def _batch_cases(case):
    return [dict(case, kind="smatrix", ny=ny, slices=nx, eta=eta) for ny, nx, eta in _batch_sizes(case)]


def _weights(case, seed):
    n_out, n_in = len(_first(case, 1)), len(_first(case, 0))
    rng = np.random.default_rng([13, seed])
    return rng.standard_normal((n_out, n_in)) + 1j * rng.standard_normal((n_out, n_in))


def prepare(case, seed):
    if case["kind"] == "channels":
        # a frequency of its own for each seed, near enough to keep the number of channels
        shift = 1e-3 * np.random.default_rng([17, seed]).random()
        count = [len(_lead(case, s)["prop"]) for s in (0, 1)]
        while [len(_lead(case, s, _k0dx(case) * (1.0 + shift))["prop"]) for s in (0, 1)] != count:
            shift *= 0.5
        return dict(case=case, k0dx=_k0dx(case) * (1.0 + shift))
    state = dict(case=case, request=_request(case))
    if case["kind"] == "batch":
        state["systs"] = [_syst(c, 1000 * seed + k) for k, c in enumerate(_batch_cases(case))]
    else:
        state["syst"] = _syst(case, seed)
    if case["kind"] == "grad":
        state["weights"] = _weights(case, seed)
    return state


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------
def _channels_out(ch):
    return [{"kx": ch[s]["kxdx" if "kxdx" in ch[s] else "kzdx"], "prop": ch[s]["ind_prop"],
             "sqrt_mu": ch[s]["sqrt_mu"]} for s in ("L", "R")]


def run(state):
    case = state["case"]
    if case["kind"] == "channels":
        ch = rgf_b200.setup_channels(case["ny"], _boundary(case), state["k0dx"], case["eps_L"], case["eps_R"])
        return {"channels": _channels_out(ch)}
    out, in_ = state["request"]
    options = {"precision": case["precision"]}
    if case["kind"] == "batch":
        return {"S": rgf_b200.cal_smatrix_RGF_batch(state["systs"], out, in_)}
    if case["kind"] == "grad":
        S, g = rgf_b200.smatrix_grad_RGF(state["syst"], out, in_, state["weights"], checkpoint=case["checkpoint"])
        return {"S": S, "g": g}
    if case["kind"] == "fields":
        S, psi = rgf_b200.fields_RGF(state["syst"], out, in_)
        return {"S": S, "psi": psi}
    call = rgf_b200.cal_smatrix_RGF if case["dim"] == 2 else rgf_b200.cal_smatrix_RGF_3D
    S, ch = call(state["syst"], out, in_, options=options)
    return {"S": S, "channels": _channels_out(ch)}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _counts(case):
    """Requested channels (out_L, out_R, in_L, in_R)."""
    p = [len(_lead(case, 0)["prop"]), len(_lead(case, 1)["prop"])]
    return {"full": (p[0], p[1], p[0], p[1]), "from_left": (p[0], p[1], p[0], 0), "transmission": (0, p[1], p[0], 0),
            "first8": (0, min(8, p[1]), min(8, p[0]), 0)}[case["request"]]


def work(case):
    if case["kind"] == "channels":
        return {"bytes": 8.0 * case["ny"] * 7, "flops": 100.0 * case["ny"]}
    if case["kind"] == "batch":
        parts = [work(c) for c in _batch_cases(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    N, L = case["nx"] * case["ny"], case["slices"]
    oL, oR, iL, iR = _counts(case)
    # per slice: the inverse, and the channel blocks of the lead it starts from
    o, i = (oL, iL) if iR else (oR, iR)
    flops = (L + 1) * (8.0 * N ** 3 + 8.0 * N * N * (o + i) + 8.0 * N * o * i)
    flops += 8.0 * N ** 3 * (1 if case["eps_L"] == case["eps_R"] else 2)
    item = 16.0 if case["eps"] in ("disks", "lossy") else 8.0
    n_out, n_in = oL + oR, iL + iR
    size = item * N * L + 16.0 * n_out * n_in
    if case["kind"] == "grad":
        flops += L * (8.0 * N * N * (n_in + n_out) + 8.0 * N * n_in * n_out)
        size += 16.0 * N * L + 16.0 * n_out * n_in
    elif case["kind"] == "fields":
        flops += L * 8.0 * N * N * n_in
        size += 16.0 * N * L * n_in
    return {"bytes": size, "flops": flops}


# ---------------------------------------------------------------------------
# the same quantities from a dense block-tridiagonal solve in complex128
# ---------------------------------------------------------------------------
def _transverse_1d(n, bc, phase):
    """Wave numbers and profiles of the transverse eigenmodes, and minus the
    second difference, of n sites."""
    m = np.arange(1, n + 1, dtype=float)
    D = 2.0 * np.eye(n, dtype=complex)
    for j in range(n - 1):
        D[j, j + 1] -= 1.0
        D[j + 1, j] -= 1.0
    if bc in ("periodic", "bloch"):
        zero = (n + 1) // 2 if n % 2 else n // 2
        k = phase / n + (m - zero) * (2 * np.pi / n)
        D[n - 1, 0] -= np.exp(1j * phase)
        D[0, n - 1] -= np.exp(-1j * phase)
        return k, np.exp(1j * np.outer(m, k)) / np.sqrt(n), D
    if bc == "Dirichlet":
        k = m * (np.pi / (n + 1))
        return k, np.sin(np.outer(m, k)) * np.sqrt(2 / (n + 1)), D
    if bc == "Neumann":
        k = (m - 1) * (np.pi / n)
        phi = np.cos(np.outer(m - 0.5, k)) * np.sqrt(2 / n)
        phi[:, 0] *= np.sqrt(0.5)
        D[0, 0] -= 1.0
        D[n - 1, n - 1] -= 1.0
        return k, phi, D
    k = (m - 0.5) * (np.pi / (n + 0.5))
    if bc == "DirichletNeumann":
        D[n - 1, n - 1] -= 1.0
        return k, np.sin(np.outer(m, k)) * np.sqrt(2 / (n + 0.5)), D
    D[0, 0] -= 1.0
    return k, np.cos(np.outer(m - 0.5, k)) * np.sqrt(2 / (n + 0.5)), D


def _transverse(case, matrices=True):
    """sin^2 of the transverse half wave numbers, profiles, A0 = minus the transverse Laplacian + 2."""
    bc = _boundary(case)
    if case["dim"] == 2:
        k, phi, D = _transverse_1d(case["ny"], case["bc"], bc if case["bc"] == "bloch" else 0.0)
        return np.sin(k / 2) ** 2, phi, D + 2 * np.eye(case["ny"])
    px, py = bc if case["bc"] == "bloch" else (0.0, 0.0)
    kx, fx, Dx = _transverse_1d(case["nx"], case["bc"], px)
    ky, fy, Dy = _transverse_1d(case["ny"], case["bc"], py)
    s2 = np.add.outer(np.sin(ky / 2) ** 2, np.sin(kx / 2) ** 2).reshape(-1)  # x fastest
    if not matrices:
        return s2, None, None
    return s2, np.kron(fy, fx), np.kron(np.eye(case["ny"]), Dx) + np.kron(Dy, np.eye(case["nx"])) + 2 * np.eye(len(s2))


def _lead(case, side, k0dx=None):
    """Longitudinal wave numbers and propagating channels (0-based) of a lead:
    4 sin^2(kx/2) = k0^2 eps - 4 sin^2(kt/2), outgoing or decaying into the lead."""
    s2 = _transverse(case, matrices=False)[0] if case["dim"] == 3 else None
    if s2 is None:
        n, bc = case["ny"], case["bc"]
        m = np.arange(1, n + 1, dtype=float)
        k = {"periodic": (m - (n + 1) // 2) if n % 2 else (m - n // 2), "Dirichlet": m, "Neumann": m - 1}.get(
            "periodic" if bc == "bloch" else bc, m - 0.5)
        k = k * {"periodic": 2 * np.pi / n, "bloch": 2 * np.pi / n, "Dirichlet": np.pi / (n + 1),
                 "Neumann": np.pi / n}.get(bc, np.pi / (n + 0.5))
        if bc == "bloch":
            k = _boundary(case) / n + k
        s2 = np.sin(k / 2) ** 2
    k0 = _k0dx(case) if k0dx is None else k0dx
    z = 0.25 * k0 ** 2 * (case["eps_L"] if side == 0 else case["eps_R"]) - s2
    prop = np.nonzero((z.real > 0) & (z.real < 1))[0]
    c = 1.0 - 2.0 * z.astype(complex)  # cos kx
    kx = np.arccos(c)
    # exp(1i kx) decays (|.| <= 1), and a propagating channel carries flux outwards
    flip = np.where(np.isin(np.arange(len(z)), prop) & (np.abs(kx.imag) < 1e-14), kx.real < 0, kx.imag < 0)
    kx = np.where(flip, -kx, kx)
    # the wave number itself, without cancellation for small z
    w = 2.0 * np.arcsin(np.sqrt(z.astype(complex)))
    near = np.abs(z) < 0.5
    kx = np.where(near, np.where(np.sign(w.imag + 1e-300) == np.sign(kx.imag + 1e-300), w, -w), kx)
    return {"kx": kx, "prop": prop, "sqrt_mu": np.sqrt(np.sin(kx[prop]))}


_EXACT_LIMIT = 4.0e5  # slices x sites: keeps the dense solve to seconds


def _wave_numbers_out(case, k0dx=None):
    leads = [_lead(case, s, k0dx) for s in (0, 1)]
    return [{"kx": None, "prop": None, "sqrt_mu": d["sqrt_mu"]} for d in leads]


def _solve(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.complex128, device=dev)  # noqa: E731
    N, L = case["nx"] * case["ny"], case["slices"]
    _, phi, A0 = _transverse(case)
    leads = [_lead(case, s) for s in (0, 1)]
    eps = np.asarray(_syst(case, seed)["epsilon"], dtype=complex).reshape((N, L), order="F")
    phi_t, A0 = t(phi), t(A0)
    G0 = [(phi_t * t(np.exp(1j * d["kx"]))[None, :]) @ phi_t.conj().T for d in leads]
    oL, oR, iL, iR = _counts(case)
    outs = [d["prop"][:n] for d, n in zip(leads, (oL, oR))]
    ins = [d["prop"][:n] for d, n in zip(leads, (iL, iR))]
    C = [t(np.sqrt(np.sin(d["kx"][o]))[:, None] * phi[:, o].conj().T) for d, o in zip(leads, outs)]
    B = [t(np.sqrt(np.sin(d["kx"][i]))[None, :] * phi[:, i]) for d, i in zip(leads, ins)]
    n_in, n_out = iL + iR, oL + oR
    k2 = _k0dx(case) ** 2
    diag = t(k2 * eps)
    g = []
    for k in range(L):
        M = A0 - torch.diag(diag[:, k])
        if k:
            M = M - g[-1]
        if k == 0:
            M = M - G0[0]
        if k == L - 1:
            M = M - G0[1]
        g.append(torch.linalg.inv(M))

    def substitute(first, last, transposed):
        """x with H x = b, b = first on slice 0 and last on the final slice (H transposed likewise)."""
        op = (lambda k: g[k].T) if transposed else (lambda k: g[k])
        r = [first if L > 1 else first + last]
        for k in range(1, L):
            r.append(op(k - 1) @ r[-1] + (last if k == L - 1 else 0))
        x = [None] * L
        for k in range(L - 1, -1, -1):
            x[k] = op(k) @ (r[k] if k == L - 1 else r[k] + x[k + 1])
        return x

    zi = lambda n: torch.zeros((N, n), dtype=torch.complex128, device=dev)  # noqa: E731
    x = substitute(torch.cat([G0[0] @ B[0], zi(iR)], 1), torch.cat([zi(iL), G0[1] @ B[1]], 1), False)
    surface = [torch.cat([B[0], zi(iR)], 1) + x[0], torch.cat([zi(iL), B[1]], 1) + x[L - 1]]
    S = -2j * torch.cat([C[s] @ (G0[s] @ surface[s]) for s in (0, 1)], 0)
    D = torch.zeros((n_out, n_in), dtype=torch.complex128, device=dev)
    for q in range(min(oL, iL)):
        D[q, q] = 1
    for q in range(min(oR, iR)):
        D[oL + q, iL + q] = 1
    S = (S - D).cpu().numpy()
    if case["kind"] == "fields":
        return S, torch.stack(x, 1).cpu().numpy()
    if case["kind"] == "grad":
        y = substitute(torch.cat([(C[0] @ G0[0]).T, zi(oR)], 1), torch.cat([zi(oL), (C[1] @ G0[1]).T], 1), True)
        W = t(_weights(case, seed))
        grad = torch.stack([((y[k] @ W) * x[k]).sum(1) for k in range(L)], 1)
        return S, (-2j * k2 * grad).cpu().numpy()
    return S, None


def exact(case, seed):
    if case["kind"] == "channels":
        return {"channels": _wave_numbers_out(case, prepare(case, seed)["k0dx"])}
    if case["kind"] == "batch":
        if sum(c["ny"] * c["slices"] for c in _batch_cases(case)) > _EXACT_LIMIT:
            return None
        return {"S": [_solve(c, 1000 * seed + k)[0] for k, c in enumerate(_batch_cases(case))]}
    if case["nx"] * case["ny"] * case["slices"] > _EXACT_LIMIT:
        return None
    S, more = _solve(case, seed)
    if case["kind"] == "grad":
        return {"S": S, "g": more}
    if case["kind"] == "fields":
        return {"S": S, "psi": more}
    return {"S": S, "channels": _wave_numbers_out(case)}
