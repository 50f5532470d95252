"""Solves of several handles on streams of their own run side by side: the default
team leaves SMs for the others, and is the team that the options can name."""
import ctypes as C
import time

import numpy as np
import pytest
import torch

from titus_b200 import Settings, SolverCSD, _lib

pytestmark = pytest.mark.gpu

# One after the other, h solves take h times as long as one; side by side about as
# long as one. Halfway in between separates the two.
CASES = [(_lib.TITUS_DLR_FIXED, 60, 20, 5, 4, 32), (_lib.TITUS_DLR_HIGH_ORDER, 60, 20, 5, 4, 32),
         (_lib.TITUS_BUG_ADAPTIVE, 90, 20, 5, 2, 64)]


@pytest.mark.parametrize("method,cells,r,npn,handles,team", CASES)
def test_side_by_side(method, cells, r, npn, handles, team):
    lib = _lib.load()
    solvers = [SolverCSD(Settings(cells + 1, cells + 1, r, "csdPhantom", nPN=npn)) for _ in range(handles)]
    streams = [torch.cuda.Stream() for _ in solvers]

    def solve(sv, stream, team_ctas=0):
        opt = sv.options(40)
        opt.team_ctas = team_ctas
        _lib.check(lib.titus_solve_device(sv.handle(), method, C.byref(opt), C.c_void_p(stream)), "titus_solve_device")

    def seconds(count):
        best = np.inf
        for _ in range(4):                      # the first makes the handles
            torch.cuda.synchronize()
            t = time.perf_counter()
            for sv, st in zip(solvers[:count], streams):
                solve(sv, st.cuda_stream)
            torch.cuda.synchronize()
            best = min(best, time.perf_counter() - t)
        return best

    def dose(sv):
        out, res = np.empty(sv.n), _lib.Result()
        res.dose = _lib.as_dp(out)
        _lib.check(lib.titus_fetch(sv.handle(), C.byref(res)), "titus_fetch")
        return out

    assert seconds(handles) < 0.5 * (1 + handles) * seconds(1)
    beside = [dose(sv) for sv in solvers]
    solve(solvers[0], None, team)
    for d in beside:
        assert np.array_equal(d, dose(solvers[0]))
