"""A job's CTA cap (cpdlp_submit's max_ctas) over LPs that go to every kind of
launch: one CTA and clusters in shared memory, tile kernels and tile clusters
(rows of more than 64 nonzeros).  How many LPs run at a time changes no result:
the capped job's solutions are the uncapped job's, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _with_long_row(lp, length):
    """lp and one more constraint over its first `length` variables."""
    from coolpdlp import generators as G
    cols = np.repeat(np.arange(lp.n), np.diff(lp.colptr))
    rows, vals = np.append(lp.rowval - 1, np.full(length, lp.m)), np.append(lp.nzval, np.ones(length))
    colptr, rowval, nzval = G.csc_from_triplets(lp.m + 1, lp.n, rows, np.append(cols, np.arange(length)), vals)
    return G.LPData(lp.m + 1, lp.n, colptr, rowval, nzval, lp.c, lp.lv, lp.uv, np.append(lp.lc, -np.inf),
                    np.append(lp.uc, 10.0 * length))


def _mix():
    from coolpdlp import generators as G
    lps = [G.random_sparse_lp(m, 2 * m, k, seed=m) for m, k in
           ((40, 4), (60, 3), (200, 5), (400, 4), (900, 5), (1500, 8), (4000, 5))]
    return lps + [_with_long_row(G.random_sparse_lp(m, 2 * m, 5, seed=m), 80) for m in (60, 300, 1600)]


@pytest.mark.parametrize("float_type", ["F64", "F32"])
def test_capped_job_gives_the_same_results(handle, float_type):
    from coolpdlp import native, _abi as A
    S = [native.LPStruct(lp.m, lp.n, lp.colptr, lp.rowval, lp.nzval, lp.c, lp.lv, lp.uv, lp.lc, lp.uc)
         for lp in _mix()]
    prm = A.default_params_py(A.ALGO_PDLP)
    prm.float_type = getattr(A, f"VAL_{float_type}")
    prm.max_kkt_passes = 1000
    prm.termination_reltol = 1e-8
    prm.power_maxiter_override = 200
    want = native.batch_solve(handle, S, prm)
    for cap in (1, 9, 40, 152):
        job = native.Job(handle, S, prm, max_ctas=cap)
        got = job.result()
        job.close()
        for k in range(len(S)):
            assert np.array_equal(got[0][k], want[0][k]) and np.array_equal(got[1][k], want[1][k]), (cap, k)
            assert got[2][k].kkt_passes == want[2][k].kkt_passes
