"""Large results reach the host by several threads and pinned buffers: the same
bytes as the plain copy, nothing written outside the k columns of a row."""
import ctypes as C
import threading

import numpy as np
import pytest

from titus_b200 import Settings, SolverCSD, _lib

pytestmark = pytest.mark.gpu


def fetch_x(solver, cap):
    res, bufs = solver._result(cap)
    X = np.full((solver.n, cap), 7.5)
    res.X = _lib.as_dp(X)
    _lib.check(_lib.load().titus_fetch(solver.handle(), C.byref(res)), "titus_fetch")
    return X, res.rank


@pytest.mark.parametrize("nx,cap", [(201, 64), (171, 80), (181, 79)])
def test_strided_rows(nx, cap):
    solver = SolverCSD(Settings(nx, nx, 7, "csdWaterBeam", nPN=5))
    res, _ = solver._result(7)
    opt = solver.options(3)
    _lib.check(_lib.load().titus_solve(solver.handle(), _lib.TITUS_DLR_FIXED, C.byref(opt), C.byref(res)), "titus_solve")
    plain, k = fetch_x(solver, 7)          # below the threaded copy's size
    assert plain.nbytes < (16 << 20) <= solver.n * cap * 8
    got = [None, None]

    def run(i):
        got[i] = fetch_x(solver, cap)[0]

    threads = [threading.Thread(target=run, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for X in got:
        assert np.array_equal(X[:, :k], plain[:, :k])
        assert np.all(X[:, k:] == 7.5)
