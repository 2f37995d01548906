"""Device memory taken while a matrix or a problem is built: rows that suit the
sliced engine badly (one of 64 entries in every 256, the others empty: slices 32
times the nonzeros) take no more than as many entries in even rows.  Measured as
the high-water mark of the device's memory pool."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

M, PER = 1 << 20, 64
USED_NOW, USED_HIGH = 7, 8  # cudaMemPoolAttrUsedMemCurrent, cudaMemPoolAttrUsedMemHigh


class Pool:
    def __init__(self):
        import torch  # noqa: F401  (loads the runtime)
        try:
            self.rt = ctypes.CDLL("libcudart.so.13")
        except OSError:
            self.rt = ctypes.CDLL("/usr/local/cuda/lib64/libcudart.so")
        self.pool = ctypes.c_void_p()
        assert self.rt.cudaDeviceGetDefaultMemPool(ctypes.byref(self.pool), 0) == 0

    def get(self, attr):
        v = ctypes.c_uint64()
        assert self.rt.cudaMemPoolGetAttribute(self.pool, attr, ctypes.byref(v)) == 0
        return v.value

    def high_water(self, f):
        zero = ctypes.c_uint64(0)
        assert self.rt.cudaMemPoolSetAttribute(self.pool, USED_HIGH, ctypes.byref(zero)) == 0
        before = self.get(USED_NOW)
        keep = f()
        high = self.get(USED_HIGH) - before
        del keep
        return high


def _csc(even):
    """M x 4096, M / 4 entries: one in every 4th row, or 64 in every 256th."""
    nnz = M // 256 * PER
    k = np.arange(nnz)
    rows = 4 * k if even else 256 * (k // PER)
    cols = (k // PER * 7 + k % PER * 61) % 4096
    import scipy.sparse as sp
    return sp.csc_matrix((1.0 + k % 5, (rows, cols)), shape=(M, 4096))


@pytest.mark.parametrize("fmt", ["CSR", "COO"])
def test_matrix_memory(handle, fmt):
    import coolpdlp as cp
    cls = {"CSR": cp.GPUSparseMatrixCSR, "COO": cp.GPUSparseMatrixCOO}[fmt]
    pool = Pool()
    even, uneven = _csc(True), _csc(False)
    cls(even, np.float64)
    a, b = (pool.high_water(lambda: cls(A, np.float64)) for A in (even, uneven))
    assert 0 < b <= 1.25 * a, (a, b)


def test_coo_holds_no_csr_beside_its_slices(handle):
    """Triplets and slices, where a CSR matrix holds the CSR and slices: a second
    row index an entry in place of the row pointer."""
    import coolpdlp as cp
    pool = Pool()
    S = _csc(True)
    held = {}
    for cls in (cp.GPUSparseMatrixCSR, cp.GPUSparseMatrixCOO):
        before = pool.get(USED_NOW)
        A = cls(S, np.float64)
        held[cls] = pool.get(USED_NOW) - before
        A.close()
    assert held[cp.GPUSparseMatrixCOO] <= held[cp.GPUSparseMatrixCSR] + 4 * S.nnz + 4096


def test_problem_memory(handle):
    from coolpdlp import native, _abi as A
    prm = A.default_params_py(A.ALGO_PDLP)
    pool = Pool()

    def build(S):
        n = 4096
        L = native.LPStruct(M, n, S.indptr + 1, S.indices + 1, S.data, np.ones(n), np.zeros(n),
                            np.ones(n), np.full(M, -np.inf), np.full(M, 1e6))
        return native.Problem(handle, L, prm)

    even, uneven = _csc(True), _csc(False)
    for S in (even, uneven):
        S.sort_indices()
    build(even)
    a, b = (pool.high_water(lambda: build(S)) for S in (even, uneven))
    assert 0 < b <= 1.25 * a, (a, b)
