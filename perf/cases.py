"""Cases that time this package through its public entry points.

Each case is one call that a user of the package makes, at the sizes of the
benchmark problems and around them:

* ``flux``       the limited second-order flux of the ordinates, on device arrays;
* ``pn``         the full-rank P_N sweep of a 2D phantom (u, dose, psi to the host);
* ``adjoint``    the dose objective of that sweep with its density and profile gradients;
* ``pn3``        the full-rank sweep of the 3D proton problem;
* ``solve``      a low-rank integrator from the reference's initial factors;
* ``resume``     a low-rank integrator continued from a mid-sweep checkpoint
                 (the ranks at which a whole solve spends nearly all of its steps);
* ``batch``      many pencil beams in one launch.

Whole solves take tens of seconds, so a pass runs the first ``steps`` energy
steps (or ``steps`` from the checkpoint). The low-rank integrators amplify
rounding over long runs (their rank decisions and truncated directions depend
on it), so the step counts stay where two summation orders agree to 1e-10 and
the outputs are the quantities that do not depend on the choice of bases: dose,
scalar flux, psi, singular values and ranks. For the same reason they have no
64-bit value apart from the algorithm itself, and ``exact`` gives none for them.
"""
import math

import numpy as np
import torch

from titus_b200 import (DoseAdjoint, Settings, Settings3D, SolveFirstCollisionSource, SolveFirstCollisionSourceDLR,
                        SolveFirstCollisionSourceDLRBUGRejection, SolveFirstCollisionSourceDLRHighOrder,
                        SolveFirstCollisionSourceDLRParallel, SolverCSD, SolverCSD3D, scalar_flux)
from titus_b200 import _lib
from titus_b200.flux import limited_flux_device

METHODS = {"fixed": _lib.TITUS_DLR_FIXED, "rk4": _lib.TITUS_DLR_HIGH_ORDER, "bug": _lib.TITUS_BUG_ADAPTIVE,
           "parallel": _lib.TITUS_PARALLEL_ADAPTIVE}
SOLVES = {"fixed": SolveFirstCollisionSourceDLR, "rk4": SolveFirstCollisionSourceDLRHighOrder,
          "bug": SolveFirstCollisionSourceDLRBUGRejection, "parallel": SolveFirstCollisionSourceDLRParallel}


def listed():
    return [
        # one sweep's flux on the 100 x 100 water-beam grid: a launch of a few microseconds, called per step
        dict(name="flux_100", kind="flux", nx=100, ny=100, q=12),
        # the flux alone on a grid larger than L2
        dict(name="flux_2048", kind="flux", nx=2048, ny=2048, q=16),
        # full-rank sweep on the 200 x 200 phantom at P29 (900 moments), and its gradients on the 100 x 100 grid
        dict(name="pn_200_P29", kind="pn", nx=200, ny=200, npn=29, steps=40),
        dict(name="adjoint_100_P21", kind="adjoint", nx=100, ny=100, npn=21, steps=40),
        # full-rank sweep of the proton problem at P13 on a 64^3 grid
        dict(name="pn3_64_P13", kind="pn3", nx=64, ny=64, nz=64, npn=13, steps=40),
        # the benchmark solve's opening (rank 40, then the ranks the beam needs) ...
        dict(name="bug_open_200_P29", kind="solve", method="bug", nx=200, ny=200, npn=29, r=80, steps=40),
        # ... and its mid-sweep steps, with either rank-adaptive integrator
        dict(name="bug_mid_200_P29", kind="resume", method="bug", nx=200, ny=200, npn=29, r=80, rank=8, steps=40),
        dict(name="parallel_mid_128_P21", kind="resume", method="parallel", nx=128, ny=128, npn=21, r=60, rank=8,
             steps=6),
        # the fixed-rank and RK4 integrators at the water-beam size and rank
        dict(name="fixed_100_P21_r20", kind="resume", method="fixed", nx=100, ny=100, npn=21, r=20, rank=20, steps=60),
        dict(name="rk4_100_P21_r20", kind="resume", method="rk4", nx=100, ny=100, npn=21, r=20, rank=20, steps=40),
        # the proton problem's low-rank solve
        dict(name="bug3_48_P13", kind="resume", method="bug", nx=48, ny=48, nz=48, npn=13, r=40, rank=6, steps=8),
        # a plan of pencil beams on the 128 x 128 phantom
        dict(name="batch_128_P21_s64", kind="batch", nx=128, ny=128, npn=21, r=60, spots=64, steps=12),
    ]


def _between(rng, lo, hi):
    """An integer of [lo, hi], uniform in its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["flux", "pn", "adjoint", "pn3", "bug", "parallel", "fixed", "rk4", "bug3", "batch"])
    if kind == "flux":
        return dict(kind="flux", nx=_between(rng, 24, 2048), ny=_between(rng, 24, 2048), q=rng.randint(3, 16))
    if kind in ("pn", "adjoint"):
        nx, ny = _between(rng, 24, 160), _between(rng, 24, 160)
        npn = _between(rng, 3, 25) if kind == "pn" else _between(rng, 3, 19)
        return dict(kind=kind, nx=nx, ny=ny, npn=npn, steps=rng.randint(12, 36))
    if kind == "pn3":
        return dict(kind="pn3", nx=rng.randint(14, 56), ny=rng.randint(14, 56), nz=rng.randint(14, 56),
                    npn=_between(rng, 3, 13), steps=rng.randint(8, 32))
    if kind == "bug3":
        return dict(kind="resume", method="bug", nx=rng.randint(18, 44), ny=rng.randint(18, 44),
                    nz=rng.randint(18, 44), npn=rng.randint(7, 13), r=rng.randint(24, 40), rank=rng.randint(3, 6),
                    steps=rng.randint(4, 8))
    if kind == "batch":
        # plans of one phantom: whether a beam's first steps amplify rounding depends on the grid and the inserts
        return dict(kind="batch", nx=128, ny=128, npn=21, r=60, spots=rng.randint(5, 63), steps=rng.randint(6, 12))
    nx, ny, npn = _between(rng, 60, 180), _between(rng, 60, 180), rng.randint(9, 27)
    if kind in ("fixed", "rk4"):
        rank = rng.randint(4, 20)
        return dict(kind="resume", method=kind, nx=min(nx, 110), ny=min(ny, 110), npn=min(npn, 21), r=rank, rank=rank,
                    steps=rng.randint(10, 40))
    if kind == "parallel":
        return dict(kind="resume", method=kind, nx=nx, ny=ny, npn=min(npn, 21), r=rng.randint(40, 80),
                    rank=rng.randint(8, 9), steps=rng.randint(3, 5))
    return dict(kind="resume", method=kind, nx=nx, ny=ny, npn=npn, r=rng.randint(40, 80), rank=rng.randint(4, 9),
                steps=rng.randint(10, 36))


# ------------------------------------------------------------------- inputs
def _solver(case, seed):
    """Solver of a phantom with a seeded entry point; the pencil-beam plan keeps the default phantom."""
    rng = np.random.default_rng(seed)
    r = case.get("r", 4)
    if "nz" in case:
        s = Settings3D(case["nx"] + 1, case["ny"] + 1, case["nz"] + 1, r=min(r, (case["npn"] + 1) ** 2),
                       nPN=case["npn"], seed=seed)
        # off-centre and anisotropic: a beam on the symmetry axis has pairs of equal singular values
        s.y0, s.z0 = (4.75 * f for f in (rng.uniform(0.8, 0.95), rng.uniform(1.05, 1.2)))
        s.sigmaZInv *= 1.5
        return SolverCSD3D(s)
    s = Settings(case["nx"] + 1, case["ny"] + 1, min(r, (case["npn"] + 1) ** 2),
                 "csdPhantom", nPN=case["npn"], **({} if case["kind"] == "batch" else {"seed": seed}))
    s.y0 = rng.uniform(0.4, 0.6)
    return SolverCSD(s)


def _checkpoint(sv, rank, seed):
    """A mid-sweep state: smooth spatial modes that decay away from the beam,
    angular modes that decay with the degree as a solve's do, singular values
    over two decades, and the uncollided beam and dose of that depth."""
    s = sv.settings
    rng = np.random.default_rng(seed)
    cell = np.arange(sv.n)
    ny = s.NCellsY
    x, y = s.xMid[cell // ny % s.NCellsX], s.yMid[cell % ny]
    L = float(s.xMid[-1])
    off = [(y - s.y0) / L]
    if "z0" in vars(s):
        off.append((s.zMid[cell // (ny * s.NCellsX)] - s.z0) / L)
    X = np.empty((sv.n, rank))
    for m in range(rank):
        f = np.exp(-x / L / rng.uniform(0.2, 0.6)) * np.cos(m * x / L + rng.uniform(0, 6))
        for k, o in enumerate(off):
            f *= np.exp(-((o - rng.uniform(-0.05, 0.05)) / rng.uniform(0.1, 0.25)) ** 2)
            f *= np.cos((m % 4 if k == 0 else m // 4) * 3.0 * o + rng.uniform(0, 6))
        X[:, m] = f
    X[sv.boundaryIdx] = 0.0
    X = np.linalg.qr(X)[0]
    degree = np.floor(np.sqrt(np.arange(sv.N)))
    W = np.linalg.qr(rng.standard_normal((sv.N, rank)) * np.exp(-0.35 * degree)[:, None])[0]
    turn = [np.linalg.qr(rng.standard_normal((rank, rank)))[0] for _ in range(2)]
    S = (turn[0] * (3e3 * 10.0 ** (-2.0 * np.arange(rank) / max(1, rank - 1)))) @ turn[1].T
    beam = np.exp(-x / (0.3 * L)) * np.exp(-sum((o / 0.05) ** 2 for o in off))
    psi = 200.0 * beam[:, None] * (sv.bc_angle / sv.bc_angle.max())[None, :]
    return dict(X=X, S=S, W=W, psi=psi, dose=20.0 * beam)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "flux":
        gen = torch.Generator("cuda").manual_seed(seed)
        rand = lambda *shape: torch.rand(shape, dtype=torch.float64, device="cuda", generator=gen)  # noqa: E731
        nx, ny, q = case["nx"], case["ny"], case["q"]
        # a smooth beam with noise of a tenth of it, directions of both signs
        i, j = torch.arange(nx, device="cuda")[:, None, None], torch.arange(ny, device="cuda")[None, :, None]
        beam = torch.exp(-3.0 * i / nx) * torch.exp(-(8.0 * (j - 0.5 * ny) / ny) ** 2)
        phi = (beam + 0.1 * rand(nx, ny, q)).contiguous()
        return dict(case=case, phi=phi, flux=torch.zeros_like(phi), ox=2.0 * rand(q) - 1.0, oz=2.0 * rand(q) - 1.0)
    sv = _solver(case, seed)
    state = dict(case=case, solver=sv)
    if kind == "batch":
        rng = np.random.default_rng(seed + 1)
        # entry points clear of the inserts' edges: a grazing beam's first steps amplify rounding by ten decades
        state["batch"] = sv.batch(list(zip(rng.uniform(2.0, 8.0, case["spots"]),
                                           rng.uniform(0.38, 0.66, case["spots"]))))
        return state
    if kind == "adjoint":
        rng = np.random.default_rng(seed + 1)
        state["weight"] = rng.uniform(0.5, 1.5, sv.n)
        state["target"] = rng.uniform(0.0, 1.0, sv.n)
    if kind == "resume":
        state["checkpoint"] = _checkpoint(sv, min(case["rank"], sv.settings.r), seed + 1)
        state["n"] = sv.nE // 4
    sv.handle()
    return state


# --------------------------------------------------------------------- run
def _padded(sigma, r):
    """Singular values at the rank cap's length: the adaptive ranks differ from input to input."""
    out = np.zeros(r)
    out[:sigma.size] = sigma
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "flux":
        return limited_flux_device(state["phi"], state["flux"], state["ox"], state["oz"], 0.02, 0.03)
    sv = state["solver"]
    if kind in ("pn", "pn3"):
        u, dose, psi = SolveFirstCollisionSource(sv, case["steps"])
        return dict(u=u, dose=dose, psi=psi)
    if kind == "adjoint":
        J, dose, grho, gprof = DoseAdjoint(sv, state["weight"], state["target"], max_steps=case["steps"])
        return dict(J=J, dose=dose, density=grho, profile=gprof)
    if kind == "batch":
        state["batch"].solve_device(_lib.TITUS_BUG_ADAPTIVE, 1, case["steps"])
        dose, rank, iterations = state["batch"].fetch()
        return dict(dose=dose, rank=rank, iterations=iterations)
    if kind == "solve":
        out = SOLVES[case["method"]](sv, max_steps=case["steps"])
        got = dict(dose=out[4], psi=out[-1], sigma=_padded(out[1], sv.settings.r),
                   flux=scalar_flux(out[0], out[1], out[3]))
        if case["method"] == "bug":
            got["ranks"] = out[5][1].astype(np.int64)
        return got
    n = state["n"]
    raw = sv.run_from(METHODS[case["method"]], state["checkpoint"], n, n + case["steps"], max_steps=case["steps"])
    out = sv.outputs(raw)
    return dict(dose=out[4], psi=out[5], sigma=_padded(out[1], sv.settings.r),
                flux=scalar_flux(out[0], out[1], out[3]), ranks=raw["rank_history"])


# -------------------------------------------------------------------- work
def work(case):
    if case["kind"] == "flux":
        words = case["nx"] * case["ny"] * case["q"]
        return dict(bytes=16.0 * words, flops=50.0 * words)
    n = case["nx"] * case["ny"] * case.get("nz", 1)
    N, q, steps = (case["npn"] + 1) ** 2, 4 if "nz" in case else 2 * case["npn"] // 3 + 2, case["steps"]
    if case["kind"] in ("pn", "pn3", "adjoint"):
        # the moment matrix read and written once a step; the operators' nonzeros per moment:
        # A_d a few, the Roe matrices dense in their eight parity classes, |Az| in its degree chains
        pairs = 3 if "nz" in case else 2
        per = 3 * pairs + (pairs - 1) * N / 8 + (case["npn"] + 1) / 3
        passes = 4 if case["kind"] == "adjoint" else 1
        return dict(bytes=steps * passes * 8.0 * (2 * n * N + 3 * n * q + 3 * n),
                    flops=steps * passes * n * N * (2.0 * per + 12 * pairs + 2 * q))
    # factors of the rank that the step keeps, read and written once a step; the products with the augmented
    # basis (Grams, K and L updates, projections)
    beams = case.get("spots", 1)
    r = case.get("rank", 4 if case["method"] == "bug" else case["r"]) if "method" in case else 4
    rows = n + N
    return dict(bytes=beams * steps * 16.0 * (rows * r + n * q + n),
                flops=beams * steps * rows * (2.0 * r) ** 2 * 24.0)


# ------------------------------------------------------------------- exact
def _dense(csr, N, device):
    rowptr, col, val = csr
    A = np.zeros((N, N))
    A[np.repeat(np.arange(N), np.diff(rowptr)), col] = val
    return torch.from_numpy(A).to(device)


def _minmod(x, y):
    lo, hi = torch.clamp(x, max=0.0), torch.clamp(x, min=0.0)
    return torch.minimum(torch.maximum(y, lo), hi)


def _slope(a, b, c):
    return _minmod(2.0 * (c - b), _minmod(0.5 * (c - a), 2.0 * (b - a)))


def _exact_flux(state):
    out = torch.zeros_like(state["phi"])
    for axis, omega, h in ((0, state["ox"], 0.02), (1, state["oz"], 0.03)):
        phi = state["phi"].transpose(0, axis)
        part = out.transpose(0, axis)[2:-2, 2:-2]
        s = [phi[k:phi.shape[0] - 4 + k, 2:-2] for k in range(5)]
        plus = (s[2] + 0.5 * _slope(s[1], s[2], s[3])) - (s[1] + 0.5 * _slope(s[0], s[1], s[2]))
        minus = (s[3] - 0.5 * _slope(s[2], s[3], s[4])) - (s[2] - 0.5 * _slope(s[1], s[2], s[3]))
        part += omega / h * torch.where(omega >= 0, plus, minus)
    return out


def _exact_sweep(sv, steps, density, profile):
    """The explicit full-rank sweep written with dense matrices; differentiable in density and profile."""
    s, dev = sv.settings, density.device
    shape = sv.psi_shape[:-1]
    nd, N = len(shape), sv.N
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    # (array axis, ordinate component, spacing, A, |A|): the arrays are (z,) x, y
    axes = [(nd - 2, 0, s.dx, sv.ops[0], sv.ops[2]), (nd - 1, 2, s.dy, sv.ops[1], sv.ops[3])]
    if nd == 3:
        axes.append((0, 1, s.dz, sv.ops3[0], sv.ops3[1]))
    axes = [(ax, t(sv.qReduced[:, comp]), h, _dense(A, N, dev), _dense(R, N, dev)) for ax, comp, h, A, R in axes]
    inner = torch.zeros(shape, dtype=torch.bool, device=dev)
    inner[(slice(1, -1),) * nd] = True
    mask = inner.reshape(-1, 1).double()
    degree = t(np.floor(np.sqrt(np.arange(N))).astype(np.int64))
    M, ang = t(sv.MReduced), t(sv.bc_angle)
    rinv = 1.0 / density
    dE = float(sv.eTrafo[1] - sv.eTrafo[0])
    u = torch.zeros(sv.n, N, dtype=torch.float64, device=dev)
    psi = torch.zeros(sv.n, sv.q, dtype=torch.float64, device=dev)
    dose = torch.zeros(sv.n, dtype=torch.float64, device=dev)

    def shift(a, ax, by):
        return torch.roll(a.reshape(shape + (-1,)), by, ax).reshape(a.shape)

    last = min(sv.nE, 1 + steps)
    for n in range(2, last + 1):
        sig = t(sv.sigma[n - 1])
        inflow = sv.bc_energy[n - 1] / sv.S[n - 1] * sv.S[n - 2] * profile[:, None] * ang
        psi = mask * psi + (1.0 - mask) * inflow
        flux = 0.0
        for ax, om, h, _, _ in axes:
            flux = flux + om / h * torch.where(om >= 0, psi - shift(psi, ax, 1), shift(psi, ax, -1) - psi)
        psi = (psi - dE * mask * flux) / (1.0 + dE * sig[0])
        v = rinv[:, None] * u
        new = u
        for ax, _, h, A, R in axes:
            lo, hi = shift(v, ax, 1), shift(v, ax, -1)
            new = new - dE / (2.0 * h) * ((hi - lo) @ A + (2.0 * v - lo - hi) @ R)
        d = sig[degree]
        u = mask * (new + dE * d * (psi @ M.T)) / (1.0 + dE * (sig[0] - d))
        half = 2.0 if n in (2, sv.nE) else 1.0
        dose = dose + dE * (u[:, 0] + mask[:, 0] * (psi @ M[0])) * float(sv.SMid[n - 2]) * rinv / half
    return u, dose, psi


def exact(case, seed):
    kind = case["kind"]
    if kind == "flux":
        return _exact_flux(prepare(case, seed))
    if kind not in ("pn", "pn3", "adjoint"):
        return None
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    sv = _solver(case, seed)
    density = torch.from_numpy(sv.density).to(dev)
    profile = torch.from_numpy(sv.bc_space).to(dev)
    if kind != "adjoint":
        with torch.no_grad():
            u, dose, psi = _exact_sweep(sv, case["steps"], density, profile)
        u *= 0.5 * math.sqrt(2.0)
        return dict(u=u, dose=dose, psi=psi.reshape(sv.psi_shape))
    rng = np.random.default_rng(seed + 1)
    weight = torch.from_numpy(rng.uniform(0.5, 1.5, sv.n)).to(dev)
    target = torch.from_numpy(rng.uniform(0.0, 1.0, sv.n)).to(dev)
    density.requires_grad_(True)
    profile.requires_grad_(True)
    _, dose, _ = _exact_sweep(sv, case["steps"], density, profile)
    J = (weight * (dose - target) ** 2).sum()
    J.backward()
    return dict(J=J.item(), dose=dose.detach(), density=density.grad, profile=profile.grad)
