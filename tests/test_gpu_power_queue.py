"""The power method of a large LP queues little beyond its last iteration: an LP
that stops by the tolerance after k iterations takes hardly longer than one that
the iteration limit stops after the same k (nothing is queued beyond a limit).
Iterations of about 0.1 ms, 10 to 20 of them; two dozen queued in vain would
take the ratio to 2."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_little_is_queued_beyond_the_last_iteration(handle):
    from coolpdlp import native, _abi as A
    rng = np.random.RandomState(8)
    n, per_col = 20000, 200
    rows = ((np.arange(n) * 7)[:, None] + np.sort(rng.choice(n, per_col, False))[None, :]) % n
    rows.sort(axis=1)
    colptr = 1 + per_col * np.arange(n + 1)
    S = native.LPStruct(n, n, colptr, rows.ravel() + 1, rng.rand(n * per_col) - 0.45, np.ones(n), np.zeros(n),
                        np.ones(n), np.full(n, -np.inf), np.ones(n))
    prm = A.default_params_py(A.ALGO_PDLP)
    prm.ruiz_iter = 0
    P = native.Problem(handle, S, prm)
    prm.power_tol_override = 1e-300
    prm.power_maxiter_override = 40
    theta = [P.spectral_norm(prm)[0] for _ in range(2)][0]

    def best(tol, limit):
        prm.power_tol_override, prm.power_maxiter_override = tol, limit
        times = []
        for _ in range(7):
            t = time.perf_counter()
            its = P.spectral_norm(prm)[1]
            times.append(time.perf_counter() - t)
        return min(times), its

    # a tolerance met within 10 to 20 iterations
    for tol in theta * theta * np.geomspace(1e-1, 1e-10, 28):
        by_tol, its = best(tol, 10**6)
        if its >= 10:
            break
    assert 10 <= its <= 20
    by_limit, same = best(1e-300, its - 1)
    assert same == its
    assert by_tol <= 1.35 * by_limit, (by_tol, by_limit, its)
