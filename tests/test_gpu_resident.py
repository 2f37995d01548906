"""LPs solved in shared memory (csrc/resident.cuh) against the Float64 oracle.

The sizes sit where the layout changes: slices of 32 rows (31, 32, 33), one
CTA or a cluster of 8 with 1,500 nonzeros and FP64 iterates, fewer ranks when
there are fewer slices than ranks, FP32 LPs of one, two and more CTAs' shared
memory, and a row of 64 nonzeros (the longest a slice holds) or 65 (the tile
kernels).  `check_every` crosses the 128-step coefficient table.

Tolerances: FP64 iterates after at most 600 steps 1e-9 of the oracle's norm
(the single-LP parity rule); FP32 solves to 1e-4 as the batch tests compare
them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _planted(m, n, rows, cols, vals, seed):
    from coolpdlp import generators as G
    st = G.Stream(seed, 91)
    c, lc, uc = G._feasible_rhs(st, rows, cols, vals, m, n, m // 2)
    colptr, rowval, nzval = G.csc_from_triplets(m, n, rows, cols, vals)
    return G.LPData(m, n, colptr, rowval, nzval, c, np.zeros(n), np.full(n, 10.0), lc, uc)


def _long_row_lp(length, seed=5):
    """40 x 200: a diagonal-like matrix whose first row has `length` nonzeros."""
    from coolpdlp import generators as G
    m, n = 40, 200
    cols = np.concatenate([np.arange(length), np.arange(n)])
    rows = np.concatenate([np.zeros(length, dtype=np.int64), 1 + np.arange(n) % (m - 1)])
    return _planted(m, n, rows, cols, G.Stream(seed, 92).normal(rows.size), seed)


def _lp(name):
    from coolpdlp import generators as G
    if name.startswith("row"):
        return _long_row_lp(int(name[3:]))
    if name.startswith("flow"):
        return G.multicommodity_flow_lp(side=int(name[4:]), K=3, seed=6)
    m, n, k = (int(v) for v in name.split("x"))
    return G.random_sparse_lp(m, n, k, seed=m + n)


def _check(handle, oracle, lp, passes, check_every, algorithm):
    from coolpdlp import native
    prm = oracle.params(algorithm, termination_reltol=0.0, max_kkt_passes=passes,
                        check_every=check_every, record_error_history=0)
    xo, yo, so = oracle.solve(lp, prm)
    S = native.LPStruct(lp.m, lp.n, lp.colptr, lp.rowval, lp.nzval, lp.c, lp.lv, lp.uv, lp.lc,
                        lp.uc)
    xs, ys, st = native.batch_solve(handle, [S, S], prm)
    assert st[0].kkt_passes == so["kkt_passes"] and st[0].termination_status == so["termination_status"]
    assert np.array_equal(xs[0], xs[1]) and np.array_equal(ys[0], ys[1])
    for a, b in ((xs[0], xo), (ys[0], yo)):
        assert np.linalg.norm(a - b) <= 1e-9 * max(1.0, np.linalg.norm(b)), lp.name


@pytest.mark.parametrize("name", ["1x3x1", "31x62x4", "32x33x5", "33x31x5", "149x300x5",
                                  "190x380x8", "255x513x6", "500x1000x5", "1300x2600x7", "row64",
                                  "row65", "flow9"])
@pytest.mark.parametrize("check_every,passes", [(100, 300), (1, 4), (257, 514)])
def test_resident_fp64(handle, oracle, name, check_every, passes):
    from coolpdlp import _abi as A
    _check(handle, oracle, _lp(name), passes, check_every, A.ALGO_PDLP)


@pytest.mark.parametrize("name", ["33x31x5", "255x513x6", "1100x2200x8", "1700x3400x8", "4000x8000x5",
                                  "row64", "row65"])
def test_resident_fp32(handle, oracle, name):
    """One CTA, then clusters of 2, 4 and 8 as the matrices outgrow it.  FP32
    stops the power method at 1%, so the step sizes differ from the oracle's and
    only a solve to 1e-4 is comparable: OPTIMAL, objective within the tolerance
    that two 1e-4 solutions have (1e-2)."""
    from coolpdlp import native, _abi as A
    lp = _lp(name)
    prm = A.default_params_py(A.ALGO_PDLP)
    xo, _, so = oracle.solve(lp, oracle.params())
    prm.float_type = A.VAL_F32
    S = native.LPStruct(lp.m, lp.n, lp.colptr, lp.rowval, lp.nzval, lp.c, lp.lv, lp.uv, lp.lc,
                        lp.uc)
    xs, ys, st = native.batch_solve(handle, [S, S], prm)
    assert so["termination_status"] == 0 and st[0].termination_status == 0
    assert np.array_equal(xs[0], xs[1]) and np.array_equal(ys[0], ys[1])
    oo = float(lp.c @ xo)
    assert abs(float(lp.c @ xs[0]) - oo) <= 1e-2 * max(1.0, abs(oo))


@pytest.mark.parametrize("name", ["33x31x5", "500x1000x5", "flow9"])
def test_resident_pdhg(handle, oracle, name):
    from coolpdlp import _abi as A
    _check(handle, oracle, _lp(name), 300, 100, A.ALGO_PDHG)
