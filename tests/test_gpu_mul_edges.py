"""mul! of the three formats at the edges of their kernels' layouts: rows of 0,
7 to 9, 16, 17 (chunks of eight), 64 and 65 nonzeros (the sliced engine's
longest row), 31 to 33 and 255 to 257 rows (slices, windows, blocks).

FP64 rows of at most 64 nonzeros are summed in column order with every product
and addition rounded: bit-identical to that sum for CSR, COO and ELL with
beta = 0.  Longer rows and FP32: n * eps of the sum of absolute products."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 7, 8, 9, 16, 17, 63, 64]


def _matrix(m, n, lengths, seed):
    from coolpdlp import generators as G
    st = G.Stream(seed, 95)
    rows = np.repeat(np.arange(m), [lengths[i % len(lengths)] for i in range(m)])
    cols = np.concatenate([np.sort(np.argsort(st.uniform(n))[:lengths[i % len(lengths)]])
                           for i in range(m)]).astype(np.int64)
    import scipy.sparse as sp
    return sp.csr_matrix((st.normal(rows.size), (rows, cols)), shape=(m, n))


@pytest.mark.parametrize("fmt", ["CSR", "COO", "ELL"])
@pytest.mark.parametrize("m,lengths", [(31, LENGTHS), (33, LENGTHS), (256, [8]), (257, LENGTHS),
                                       (1000, [3, 4]), (40, LENGTHS + [65, 300])])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_mul_edges(handle, fmt, m, lengths, dtype):
    import coolpdlp as cp
    import torch
    n = 400
    A = _matrix(m, n, lengths, seed=m + len(lengths))
    M = {"CSR": cp.GPUSparseMatrixCSR, "COO": cp.GPUSparseMatrixCOO, "ELL": cp.GPUSparseMatrixELL}[fmt]
    G = M(A.tocsc(), dtype)
    rng = np.random.RandomState(m)
    b, c0 = rng.randn(n).astype(dtype), rng.randn(m).astype(dtype)
    V = A.data.astype(dtype)
    for alpha, beta in ((1.0, 0.0), (-0.5, 2.0)):
        c = torch.from_numpy(c0 if beta else np.full(m, np.nan, dtype)).cuda()
        G.mul(c, torch.from_numpy(b).cuda(), alpha, beta)
        got = c.cpu().numpy()
        for i in range(m):
            lo, hi = A.indptr[i], A.indptr[i + 1]
            p = V[lo:hi] * b[A.indices[lo:hi]]
            s = dtype(0)
            for q in p:
                s = s + q
            want = dtype(alpha) * s + (dtype(beta) * c0[i] if beta else dtype(0))
            if beta == 0.0 and dtype == np.float64 and (hi - lo <= 64 or fmt == "ELL"):
                assert got[i] == want, (i, hi - lo)
            else:
                tol = (hi - lo + 4) * np.finfo(dtype).eps * (np.abs(p).sum() + abs(beta * c0[i]) + 1e-30)
                assert abs(got[i] - want) <= tol, (i, hi - lo, got[i], want)
