"""The sliced step engine (csrc/sell.cuh) against the tile engine and the
Float64 oracle.

It runs where no tile size is pinned; `tile_nnz` = 128, the tile size that the
library picks at these sizes, pins the tile engine.  FP32: the same products
and sums in the same order, so the iterates are bit-identical.  FP64: fused
operations, iterates after 50 steps within 1e-9 of the oracle's (the step
parity rule).  The row lengths sit at the edges of the layout: empty rows, 64
(the longest row of a slice), 65 and 128 (one piece), 129 and 700 (several
pieces), and the row counts at the edges of slices (32) and windows (256)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lp(m, n, long_rows, seed):
    """m x n, about 4 entries a column in rows 3.., row 2 empty, and rows of the
    given lengths in front (they also keep the LP off the resident kernels)."""
    from coolpdlp import generators as G
    st = G.Stream(seed, 93)
    rows, cols = [], []
    for i, length in enumerate(long_rows):
        rows.append(np.full(length, i, dtype=np.int64))
        cols.append(np.sort(np.argsort(st.uniform(n))[:length]))
    lo = len(long_rows) + 1  # row len(long_rows) stays empty
    r = lo + (np.arange(4 * n) * 7 + st.integers(4 * n, 0, 3)) % max(m - lo, 1)
    c = np.repeat(np.arange(n), 4)
    keep = np.unique(c * m + r, return_index=True)[1]
    rows.append(r[keep])
    cols.append(c[keep])
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    vals = st.normal(rows.size)
    c, lc, uc = G._feasible_rhs(st, rows, cols, vals, m, n, m // 2)
    colptr, rowval, nzval = G.csc_from_triplets(m, n, rows, cols, vals)
    return G.LPData(m, n, colptr, rowval, nzval, c, np.zeros(n), np.full(n, 10.0), lc, uc)


CASES = [(70, 800, (64, 65)), (255, 1000, (128, 129)), (2048, 8192, (700, 66)),
         (2049, 8200, (65, 64, 700)), (4700, 16400, (1200,))]


def _steps(handle, lp, prm, steps):
    from coolpdlp import native, _abi as A
    S = native.LPStruct(lp.m, lp.n, lp.colptr, lp.rowval, lp.nzval, lp.c, lp.lv, lp.uv, lp.lc,
                        lp.uc)
    st = native.State(native.Problem(handle, S, prm), prm, np.linspace(0, 1, lp.n),
                      np.linspace(-1, 1, lp.m))
    st.step(steps)
    return [v for which in (A.VEC_SOL, A.VEC_SOL_AVG) for v in st.vectors(which)]


@pytest.mark.parametrize("m,n,long_rows", CASES)
def test_sliced_fp32_is_the_tile_engines_bits(handle, m, n, long_rows):
    from coolpdlp import native, _abi as A
    lp = _lp(m, n, long_rows, seed=m + n)
    prm = A.default_params_py(A.ALGO_PDLP)
    prm.float_type = A.VAL_F32
    pinned = native.copy_params(prm)
    pinned.tile_nnz = 128
    for a, b in zip(_steps(handle, lp, prm, 50), _steps(handle, lp, pinned, 50)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("m,n,long_rows", CASES)
def test_sliced_fp64_against_oracle(handle, oracle, m, n, long_rows):
    from coolpdlp import _abi as A
    lp = _lp(m, n, long_rows, seed=m + n)
    prm = oracle.params()
    S = oracle.OracleState(lp, prm, np.linspace(0, 1, lp.n), np.linspace(-1, 1, lp.m))
    S.step(50)
    want = [v for which in (A.VEC_SOL, A.VEC_SOL_AVG) for v in S.vectors(which)]
    for a, b in zip(_steps(handle, lp, prm, 50), want):
        assert np.max(np.abs(a - b)) <= 1e-9 * max(1.0, np.max(np.abs(b)))
    S.close()


@pytest.mark.parametrize("side,K", [(3, 2), (9, 3), (12, 70)])
def test_sliced_narrow_is_the_tile_engines_bits(handle, side, K):
    """+-1 storage (signs in the indices): flow LPs, capacity rows of K entries
    (70: long pieces)."""
    from coolpdlp import generators as G, native, _abi as A
    lp = G.multicommodity_flow_lp(side=side, K=K, seed=side)
    prm = A.default_params_py(A.ALGO_PDLP)
    prm.float_type = A.VAL_F32
    pinned = native.copy_params(prm)
    pinned.tile_nnz = 128
    for a, b in zip(_steps(handle, lp, prm, 50), _steps(handle, lp, pinned, 50)):
        assert np.array_equal(a, b)
