"""Low-rank energy steps at ranks, row counts and team sizes around the edges of
the kernels' 8 x 8 blocks, row tiles and reduction rules, against the FP64 oracle.

The state is an oracle state whose factors are replaced by random orthonormal
ones and an S of condition 2, so that a step does not amplify rounding by its
own small singular values: what is left is the range finder, whose certified
condition (1e5) times the unit rounding times a few dozen rows stays below 1e-9
in the worst case and 1e-12 in practice. TOL is the other parity tests' 1e-10.
"""
import numpy as np
import pytest

from oracle.settings import Settings as OSettings
from oracle.solver import SolverCSD as OSolver
from oracle.solver import solve_dlr_bug, solve_dlr_fixed, solve_dlr_high_order, solve_dlr_parallel
from titus_b200 import Settings, SolverCSD, _lib

pytestmark = pytest.mark.gpu
TOL = 1e-10
RUN = {"fixed": (solve_dlr_fixed, _lib.TITUS_DLR_FIXED), "rk4": (solve_dlr_high_order, _lib.TITUS_DLR_HIGH_ORDER),
       "bug": (solve_dlr_bug, _lib.TITUS_BUG_ADAPTIVE), "parallel": (solve_dlr_parallel, _lib.TITUS_PARALLEL_ADAPTIVE)}


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def check(method, nx, npn, r, k, team, steps):
    fn, mid = RUN[method]

    def oracle():
        return OSolver(OSettings(nx, nx, r, "csdWaterBeam", nPN=npn))

    st = dict(solve_dlr_fixed(OSolver(OSettings(nx, nx, min(r, 8), "csdWaterBeam", nPN=npn)), max_steps=4,
                              return_state=True))
    rng = np.random.default_rng(1000 * k + team)
    n, N = (nx - 1) ** 2, (npn + 1) ** 2
    i, j = np.divmod(np.arange(n), nx - 1)
    X = rng.standard_normal((n, k))
    X[(i == 0) | (j == 0) | (i == nx - 2) | (j == nx - 2)] = 0.0
    st["X"] = np.linalg.qr(X)[0]
    st["W"] = np.linalg.qr(rng.standard_normal((N, k)))[0]
    U, V = (np.linalg.qr(rng.standard_normal((k, k)))[0] for _ in range(2))
    st["S"] = U @ np.diag(np.linspace(1.0, 0.5, k)) @ V
    n0 = st["n_next"]
    ref = fn(oracle(), max_steps=steps, state=dict(st), n_begin=n0, return_state=True)
    g = SolverCSD(Settings(nx, nx, r, "csdWaterBeam", nPN=npn), team_ctas=team)
    if method == "bug":
        got = g.run_from(mid, st, n0, g.nE, max_steps=steps)
    else:
        got = g.run_from(mid, st, n0, n0 + steps - 1)
    assert got["S"].shape == ref["S"].shape
    assert rel(got["dose"], ref["dose"]) <= TOL
    assert rel(got["psi"].ravel(), ref["psi"].ravel()) <= TOL
    assert rel(got["X"] @ got["S"] @ got["W"].T, ref["X"] @ ref["S"] @ ref["W"].T) <= TOL


@pytest.mark.parametrize("method", ["fixed", "rk4"])
@pytest.mark.parametrize("k,team", [(1, 1), (7, 16), (8, 17), (9, 0), (16, 13), (17, 14), (23, 40), (24, 0)])
def test_fixed_rank(method, k, team):
    check(method, 24, 5, k, k, team, 2)


@pytest.mark.parametrize("k,team", [(1, 1), (7, 64), (8, 3), (9, 0), (15, 17), (17, 100), (20, 0)])
def test_rank_adaptive(k, team):
    check("bug", 24, 9, 80, k, team, 1)   # the rank may double


@pytest.mark.parametrize("k,team", [(3, 0), (8, 17), (13, 0), (20, 100)])
def test_parallel(k, team):
    check("parallel", 24, 9, 80, k, team, 1)
