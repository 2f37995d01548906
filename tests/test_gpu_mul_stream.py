"""mul! after work that is still pending on a torch stream of the caller's: the
product reads what that work writes, for b and (beta != 0) for c, and torch work
queued after the call sees the result."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", ["CSR", "COO", "ELL"])
@pytest.mark.parametrize("side_stream", [False, True])
def test_mul_waits_for_the_callers_stream(handle, fmt, side_stream):
    import coolpdlp as cp
    import scipy.sparse as sp
    import torch
    rng = np.random.RandomState(5)
    m, n = 500, 700
    S = sp.random(m, n, 0.01, random_state=rng, format="csc")
    A = {"CSR": cp.GPUSparseMatrixCSR, "COO": cp.GPUSparseMatrixCOO, "ELL": cp.GPUSparseMatrixELL}[fmt](S, np.float64)
    big = torch.randn(4096, 4096, device="cuda")
    xs = [torch.from_numpy(rng.randn(n)).cuda() for _ in range(3)]
    cs = [torch.from_numpy(rng.randn(m)).cuda() for _ in range(3)]
    stream = torch.cuda.Stream() if side_stream else torch.cuda.default_stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        b, c = torch.zeros(n, dtype=torch.float64, device="cuda"), torch.zeros(m, dtype=torch.float64, device="cuda")
        for x, c0 in zip(xs, cs):
            y = big
            for _ in range(20):  # some milliseconds
                y = (y @ big) * 1e-2
            b.copy_(x)
            c.copy_(c0)
            A.mul(c, b, 2.0, -0.5)
            got = (c + 0.0).cpu().numpy()
            want = 2.0 * (S @ x.cpu().numpy()) - 0.5 * c0.cpu().numpy()
            assert np.max(np.abs(got - want)) <= 1e-12 * max(1.0, np.max(np.abs(want)))
