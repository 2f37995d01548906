"""A batched LP's time limit and time_elapsed count its steps and checks, not its
power method, whether it is solved in shared memory or (a row of more than 64
nonzeros) by the tile kernels: 20,000 power iterations take at least 50 ms, the
20 steps after them a few ms, and the limit lies between."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,row", [(1000, 0), (60, 0), (60, 80)])
def test_time_limit_excludes_the_power_method(handle, m, row):
    from coolpdlp import generators as G, native, _abi as A
    lp = G.random_sparse_lp(m, 2 * m, 5, seed=m)
    if row:
        cols = np.append(np.repeat(np.arange(lp.n), np.diff(lp.colptr)), np.arange(row))
        rows, vals = np.append(lp.rowval - 1, np.full(row, m)), np.append(lp.nzval, np.ones(row))
        colptr, rowval, nzval = G.csc_from_triplets(m + 1, lp.n, rows, cols, vals)
        lp = G.LPData(m + 1, lp.n, colptr, rowval, nzval, lp.c, lp.lv, lp.uv, np.append(lp.lc, -np.inf),
                      np.append(lp.uc, 10.0 * row))
    prm = A.default_params_py(A.ALGO_PDLP)
    prm.termination_reltol = 0.0
    prm.check_every = 1
    prm.max_kkt_passes = 20
    prm.time_limit = 0.02
    prm.power_maxiter_override = 20000
    prm.power_tol_override = 1e-300
    S = native.LPStruct(lp.m, lp.n, lp.colptr, lp.rowval, lp.nzval, lp.c, lp.lv, lp.uv, lp.lc, lp.uc)
    for _ in range(2):  # (the first call loads the kernels)
        st = native.batch_solve(handle, [S], prm)[2][0]
    assert st.power_iterations == 20001
    assert st.termination_status == A.ITERATION_LIMIT and st.kkt_passes == 20
    assert 0.0 < st.time_elapsed < 0.02
