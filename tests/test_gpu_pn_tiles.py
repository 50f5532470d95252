"""The full-rank P_N step kernels (pn_tiles.cuh) at the edges of their tiles,
against a plain torch FP64 restatement of the sweep with dense matrices.

Both kernels run: the tiled one above about 1e7 nonzeros over all cells, the
small one below. The cases hold patches that the grid cuts on every axis, more
ordinates than one in-scattering chunk (16) takes, moment classes that are not
whole tiles, and operators without the P_N structure: one dense class larger
than a column group, and a pattern without classes. The scheme is linear and
explicit (a few steps of O(N) products), so results agree to a small multiple
of N * 2^-53; 1e-12 leaves a factor of ten at N = 484.
"""
import numpy as np
import pytest
import torch

from titus_b200 import DoseAdjoint, Settings, Settings3D, SolveFirstCollisionSource, SolverCSD, SolverCSD3D
from titus_b200 import physics as ph

pytestmark = pytest.mark.gpu
TOL = 1e-12


def dense(csr, N):
    rowptr, col, val = csr
    A = np.zeros((N, N))
    A[np.repeat(np.arange(N), np.diff(rowptr)), col] = val
    return torch.from_numpy(A).cuda()


def sweep(sv, steps, density, profile):
    s, N = sv.settings, sv.N
    shape = sv.psi_shape[:-1]
    nd = len(shape)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    axes = [(nd - 2, 0, s.dx, 0, 2), (nd - 1, 2, s.dy, 1, 3)]
    axes = [(ax, t(sv.qReduced[:, c]), h, dense(sv.ops[i], N), dense(sv.ops[j], N)) for ax, c, h, i, j in axes]
    if nd == 3:
        axes.append((0, t(sv.qReduced[:, 1]), s.dz, dense(sv.ops3[0], N), dense(sv.ops3[1], N)))
    inner = torch.zeros(shape, dtype=torch.bool, device="cuda")
    inner[(slice(1, -1),) * nd] = True
    mask = inner.reshape(-1, 1).double()
    l = t(np.floor(np.sqrt(np.arange(N))).astype(np.int64))
    M, ang = t(sv.MReduced), t(sv.bc_angle)
    rinv = 1.0 / density
    dE = float(sv.eTrafo[1] - sv.eTrafo[0])
    shift = lambda a, ax, by: torch.roll(a.reshape(shape + (-1,)), by, ax).reshape(a.shape)  # noqa: E731
    u = torch.zeros(sv.n, N, dtype=torch.float64, device="cuda")
    psi = torch.zeros(sv.n, sv.q, dtype=torch.float64, device="cuda")
    dose = torch.zeros(sv.n, dtype=torch.float64, device="cuda")
    for n in range(2, 2 + steps):
        sig = t(sv.sigma[n - 1])
        inflow = sv.bc_energy[n - 1] / sv.S[n - 1] * sv.S[n - 2] * profile[:, None] * ang
        psi = mask * psi + (1 - mask) * inflow
        flux = sum(om / h * torch.where(om >= 0, psi - shift(psi, ax, 1), shift(psi, ax, -1) - psi)
                   for ax, om, h, _, _ in axes)
        psi = (psi - dE * mask * flux) / (1 + dE * sig[0])
        v = rinv[:, None] * u
        new = u
        for ax, _, h, A, R in axes:
            lo, hi = shift(v, ax, 1), shift(v, ax, -1)
            new = new - dE / (2 * h) * ((hi - lo) @ A + (2 * v - lo - hi) @ R)
        d = sig[l]
        u = mask * (new + dE * d * (psi @ M.T)) / (1 + dE * (sig[0] - d))
        half = 2.0 if n in (2, sv.nE) else 1.0
        dose = dose + dE * (u[:, 0] + mask[:, 0] * (psi @ M[0])) * float(sv.SMid[n - 2]) * rinv / half
    return u, dose, psi


def random_ops(sv, kind, seed=3):
    """Operators of the moment system's size without its structure (spectral radius below 1)."""
    rng = np.random.default_rng(seed)
    N = sv.N
    out = []
    for d in range(4):
        A = rng.standard_normal((N, N)) / (2 * np.sqrt(N))
        if kind == "sparse":
            A *= rng.random((N, N)) < 3.0 / N
        out.append(ph.to_csr(A))
    sv.ops = out


def solver2d(nx, ny, npn, widen=1.0, ops=None):
    s = Settings(nx + 1, ny + 1, 4, "csdPhantom", nPN=npn, seed=11)
    s.sigmaO1Inv /= widen
    s.sigmaO3Inv /= widen
    s.y0 = 0.43
    sv = SolverCSD(s)
    if ops:
        random_ops(sv, ops)
    return sv


def rel(a, b):
    b = b.detach().cpu().numpy().reshape(a.shape) if isinstance(b, torch.Tensor) else b
    return np.linalg.norm(a - b) / np.linalg.norm(b)


CASES_2D = [(43, 75, 13, 1.0, None), (61, 37, 21, 1.0, None), (67, 70, 13, 16.0, None), (9, 300, 13, 1.0, None),
            (24, 21, 7, 1.0, None), (3, 19, 5, 1.0, None), (13, 11, 5, 100.0, None), (40, 37, 13, 1.0, "dense"),
            (90, 120, 7, 1.0, "dense"), (120, 113, 13, 1.0, "sparse"), (12, 9, 9, 1.0, "sparse")]


@pytest.mark.parametrize("nx,ny,npn,widen,ops", CASES_2D)
def test_step_2d(nx, ny, npn, widen, ops):
    sv = solver2d(nx, ny, npn, widen, ops)
    if widen > 1.0:
        assert sv.q > 16
    u, dose, psi = SolveFirstCollisionSource(sv, max_steps=6)
    with torch.no_grad():
        ref = sweep(sv, 6, torch.from_numpy(sv.density).cuda(), torch.from_numpy(sv.bc_space).cuda())
    assert rel(u, 0.5 * np.sqrt(2.0) * ref[0]) <= TOL
    assert rel(dose, ref[1]) <= TOL
    assert rel(psi, ref[2]) <= TOL


@pytest.mark.parametrize("nx,ny,npn,widen,ops", [CASES_2D[0], CASES_2D[4], CASES_2D[6], CASES_2D[7], CASES_2D[10]])
def test_adjoint_2d(nx, ny, npn, widen, ops):
    sv = solver2d(nx, ny, npn, widen, ops)
    rng = np.random.default_rng(5)
    w, t = rng.uniform(0.5, 1.5, sv.n), rng.uniform(0.0, 1.0, sv.n)
    J, dose, grho, gprof = DoseAdjoint(sv, w, t, checkpoint_every=2, max_steps=5)
    density = torch.from_numpy(sv.density).cuda().requires_grad_(True)
    profile = torch.from_numpy(sv.bc_space).cuda().requires_grad_(True)
    _, d, _ = sweep(sv, 5, density, profile)
    Jr = (torch.from_numpy(w).cuda() * (d - torch.from_numpy(t).cuda()) ** 2).sum()
    Jr.backward()
    assert abs(J - Jr.item()) <= TOL * abs(Jr.item())
    assert rel(dose, d) <= TOL and rel(grho, density.grad) <= TOL and rel(gprof, profile.grad) <= TOL


@pytest.mark.parametrize("nx,ny,nz,npn", [(15, 21, 18, 9), (9, 34, 11, 13), (7, 10, 6, 5), (30, 28, 23, 5)])
def test_step_3d(nx, ny, nz, npn):
    s = Settings3D(nx + 1, ny + 1, nz + 1, r=4, nPN=npn, seed=7)
    s.y0, s.z0 = 4.2, 5.1
    sv = SolverCSD3D(s)
    u, dose, psi = SolveFirstCollisionSource(sv, max_steps=6)
    with torch.no_grad():
        ref = sweep(sv, 6, torch.from_numpy(sv.density).cuda(), torch.from_numpy(sv.bc_space).cuda())
    assert rel(u, 0.5 * np.sqrt(2.0) * ref[0]) <= TOL
    assert rel(dose, ref[1]) <= TOL
    assert rel(psi, ref[2]) <= TOL


def test_adjoint_without_entries_in_a_column_group():
    """Operators that hold nothing outside the first 60 of 196 moments: the second column group of the tiled
    kernel (13 of its 25 output tiles) has no chunk in the adjoint, and its columns decay by the collision alone."""
    sv = solver2d(34, 34, 13)
    rng = np.random.default_rng(8)
    ops = []
    for _ in range(4):
        A = np.zeros((sv.N, sv.N))
        A[:60, :60] = rng.standard_normal((60, 60)) / (2 * np.sqrt(60))
        ops.append(ph.to_csr(A))
    sv.ops = ops
    nnz = sum(len(v) for _, _, v in ops)
    assert 32 * 32 * nnz > 10**7               # beyond the small kernel's range
    w, t = rng.uniform(0.5, 1.5, sv.n), rng.uniform(0.0, 1.0, sv.n)
    J, dose, grho, gprof = DoseAdjoint(sv, w, t, checkpoint_every=2, max_steps=5)
    density = torch.from_numpy(sv.density).cuda().requires_grad_(True)
    profile = torch.from_numpy(sv.bc_space).cuda().requires_grad_(True)
    _, d, _ = sweep(sv, 5, density, profile)
    Jr = (torch.from_numpy(w).cuda() * (d - torch.from_numpy(t).cuda()) ** 2).sum()
    Jr.backward()
    assert abs(J - Jr.item()) <= TOL * abs(Jr.item())
    assert rel(dose, d) <= TOL and rel(grho, density.grad) <= TOL and rel(gprof, profile.grad) <= TOL


@pytest.mark.parametrize("nx,ny,npn,ldu,fours", [(80, 71, 3, 16, 4), (61, 60, 5, 48, 2)])
def test_small_kernel_with_several_fours(nx, ny, npn, ldu, fours):
    """The small kernel's CTAs of several fours of cells, the last one cut: forward and adjoint."""
    sv = solver2d(nx, ny, npn)
    cells = (nx - 2) * (ny - 2)
    assert cells * sum(len(v) for _, _, v in sv.ops) < 5 * 10**6     # well inside its range
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    f = 128 // ldu
    while f > 1 and cells < 2 * sms * 4 * f:
        f -= 1
    assert f == fours and cells % (4 * fours)
    with torch.no_grad():
        ref = sweep(sv, 6, torch.tensor(sv.density).cuda(), torch.tensor(sv.bc_space).cuda())
    u, dose, psi = SolveFirstCollisionSource(sv, max_steps=6)
    assert rel(u, 0.5 * np.sqrt(2.0) * ref[0]) <= TOL and rel(dose, ref[1]) <= TOL and rel(psi, ref[2]) <= TOL
    rng = np.random.default_rng(9)
    w, t = rng.uniform(0.5, 1.5, sv.n), rng.uniform(0.0, 1.0, sv.n)
    J, dose, grho, gprof = DoseAdjoint(sv, w, t, checkpoint_every=2, max_steps=5)
    density = torch.tensor(sv.density).cuda().requires_grad_(True)
    profile = torch.tensor(sv.bc_space).cuda().requires_grad_(True)
    _, d, _ = sweep(sv, 5, density, profile)
    Jr = (torch.from_numpy(w).cuda() * (d - torch.from_numpy(t).cuda()) ** 2).sum()
    Jr.backward()
    assert abs(J - Jr.item()) <= TOL * abs(Jr.item())
    assert rel(dose, d) <= TOL and rel(grho, density.grad) <= TOL and rel(gprof, profile.grad) <= TOL
