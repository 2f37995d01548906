"""One matrix, two handles, two threads: products of rows in several pieces (600
to 9,000 nonzeros), whose scratch belongs to one product at a time.  Every
product has the bits of the same product alone."""
import threading
from ctypes import c_void_p

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt,dtype", [("COO", np.float64), ("COO", np.float32), ("CSR", np.float64),
                                       ("CSR", np.float32), ("ELL", np.float64)])
def test_products_on_two_handles_at_a_time(handle, fmt, dtype):
    import coolpdlp as cp
    from coolpdlp import native
    import scipy.sparse as sp
    import torch
    rng = np.random.RandomState(3)
    m, n = 300, 10000
    lengths = np.where(np.arange(m) % 3 == 0, rng.randint(600, 9000, m), rng.randint(0, 9, m))
    cols = np.concatenate([np.sort(rng.permutation(n)[:k]) for k in lengths])
    S = sp.csr_matrix((rng.randn(cols.size), (np.repeat(np.arange(m), lengths), cols)), shape=(m, n))
    A = {"CSR": cp.GPUSparseMatrixCSR, "COO": cp.GPUSparseMatrixCOO, "ELL": cp.GPUSparseMatrixELL}[fmt](S.tocsc(), dtype)
    bs = [torch.from_numpy(rng.randn(n).astype(dtype)).cuda() for _ in range(2)]
    want = [A.mul(torch.zeros(m, dtype=b.dtype, device="cuda"), b).clone() for b in bs]
    torch.cuda.synchronize()
    wrong = [None, None]

    def work(k):
        h = native.Handle(0)
        cs = [torch.zeros(m, dtype=bs[k].dtype, device="cuda") for _ in range(4)]
        torch.cuda.current_stream().synchronize()
        bad = 0
        for r in range(400):
            c = cs[r % 4]
            h.check(h.lib.cpdlp_spmv(h.h, A.ptr, c_void_p(bs[k].data_ptr()), c_void_p(c.data_ptr()), 1.0, 0.0))
            bad += not np.array_equal(c.cpu().numpy(), want[k].cpu().numpy())
        h.close()
        wrong[k] = bad

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert wrong == [0, 0]
