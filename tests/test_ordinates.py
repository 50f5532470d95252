"""The largest numbers of reduced ordinates: wide beams up to the limit of 24 through
the low-rank kernels against the FP64 oracle, refused beyond it."""
import os

import numpy as np
import pytest

from oracle.settings import Settings as OSettings
from oracle.solver import SolverCSD as OSolver
from oracle.solver import solve_dlr_bug, solve_dlr_fixed, solve_dlr_high_order
from titus_b200 import Settings, SolverCSD, _lib

TOL = 1e-10      # the other parity tests'
RUN = {"fixed": (solve_dlr_fixed, _lib.TITUS_DLR_FIXED), "rk4": (solve_dlr_high_order, _lib.TITUS_DLR_HIGH_ORDER),
       "bug": (solve_dlr_bug, _lib.TITUS_BUG_ADAPTIVE)}


def widened(cls, npn, widen, r=4):
    s = cls(24, 24, r, "csdWaterBeam", nPN=npn)
    s.sigmaO1Inv /= widen
    s.sigmaO3Inv /= widen
    return s


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.skipif(not os.path.exists(_lib.LIB_PATH), reason="libtitus.so not built")
def test_beyond_the_limit():
    solver = SolverCSD(widened(Settings, 7, 100.0))
    assert solver.q == 32 and _lib.load().titus_max_ordinates() == 24
    with pytest.raises(RuntimeError, match="n_ordinates 32 > 24"):
        solver.handle()


@pytest.mark.gpu
@pytest.mark.parametrize("method", sorted(RUN))
@pytest.mark.parametrize("npn,widen,q", [(5, 60.0, 12), (5, 80.0, 20), (5, 140.0, 24), (7, 80.0, 24)])
def test_up_to_the_limit(method, npn, widen, q):
    fn, mid = RUN[method]
    k, steps = 6, 2
    r = k if method != "bug" else 32          # a cap within the 36 moments
    st = dict(solve_dlr_fixed(OSolver(widened(OSettings, npn, widen, k)), max_steps=4, return_state=True))
    rng = np.random.default_rng(q)
    i, j = np.divmod(np.arange(23 * 23), 23)
    X = rng.standard_normal((23 * 23, k))
    X[(i == 0) | (j == 0) | (i == 22) | (j == 22)] = 0.0
    st["X"] = np.linalg.qr(X)[0]
    st["W"] = np.linalg.qr(rng.standard_normal(((npn + 1) ** 2, k)))[0]
    U, V = (np.linalg.qr(rng.standard_normal((k, k)))[0] for _ in range(2))
    st["S"] = U @ np.diag(np.linspace(1.0, 0.5, k)) @ V
    n0 = st["n_next"]
    ref = fn(OSolver(widened(OSettings, npn, widen, r)), max_steps=steps, state=dict(st), n_begin=n0, return_state=True)
    g = SolverCSD(widened(Settings, npn, widen, r))
    assert g.q == q
    if method == "bug":
        got = g.run_from(mid, st, n0, g.nE, max_steps=steps)
    else:
        got = g.run_from(mid, st, n0, n0 + steps - 1)
    assert got["S"].shape == ref["S"].shape
    assert rel(got["dose"], ref["dose"]) <= TOL
    assert rel(got["psi"].ravel(), ref["psi"].ravel()) <= TOL
    assert rel(got["X"] @ got["S"] @ got["W"].T, ref["X"] @ ref["S"] @ ref["W"].T) <= TOL
