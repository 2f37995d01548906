"""A single LP on the resident kernels (csrc/resident_single.cu): blocks of steps
whose length is odd, one, or more than the 128-step coefficient table, step counts
that leave single tile steps over, and a power method that takes more than one
launch (1,024 iterations each), on groups of 1, 2, 4 and 8 CTAs (as many as the
smaller side has slices of 32 rows).

Tolerances: FP64 iterates 1e-9 of the oracle's norm (the single-LP parity rule).
FP32 iterates are compared with the tile engine's: the step size agrees to FP64
rounding, the row sums are the same, and 300 steps of FP32 rounding of
nonexpansive steps stay within 300 * eps = 4e-5 of the norm.  The norm of A: the
gap to the second singular value closes within 3,000 iterations to 1e-9."""
import numpy as np
import pytest

from test_gpu_resident import _lp

pytestmark = pytest.mark.gpu


def _struct(lp):
    from coolpdlp import native
    return native.LPStruct(lp.m, lp.n, lp.colptr, lp.rowval, lp.nzval, lp.c, lp.lv, lp.uv, lp.lc, lp.uc)


def _state(handle, lp, prm):
    from coolpdlp import native
    P = native.Problem(handle, _struct(lp), prm)
    return native.State(P, prm, np.linspace(0, 1, lp.n), np.linspace(-1, 1, lp.m)), P.layout()["A"]


FP64 = [("1x3x1", 1), ("31x62x4", 1), ("33x31x5", 1), ("62x400x5", 2), ("100x500x6", 4), ("255x513x6", 8),
        ("500x1000x5", 8), ("row64", 1), ("flow9", 1)]


@pytest.mark.parametrize("name,ctas", FP64)
@pytest.mark.parametrize("check_every,steps", [(1, 5), (101, 303), (101, 250), (257, 514), (100, 99)])
def test_blocks_fp64(handle, oracle, name, ctas, check_every, steps):
    from coolpdlp import _abi as A
    lp = _lp(name)
    prm = oracle.params(check_every=check_every)
    st, lay = _state(handle, lp, prm)
    if name != "flow9":
        assert (lay["engine"], lay["resident_ctas"]) == ("resident", ctas)
    S = oracle.OracleState(lp, prm, np.linspace(0, 1, lp.n), np.linspace(-1, 1, lp.m))
    st.step(steps)
    S.step(steps)
    for which in (A.VEC_SOL, A.VEC_SOL_LAST, A.VEC_SOL_AVG):
        for a, b in zip(st.vectors(which), S.vectors(which)):
            assert np.linalg.norm(a - b) <= 1e-9 * max(1.0, np.linalg.norm(b))
    S.close()


@pytest.mark.parametrize("algorithm", ["PDLP", "PDHG"])
@pytest.mark.parametrize("name", ["33x31x5", "62x400x5", "255x513x6"])
def test_checks_of_a_block(handle, oracle, name, algorithm):
    """The KKT errors that come with a block are those of its iterates (which no
    restart replaces here)."""
    from coolpdlp import _abi as A
    lp = _lp(name)
    prm = oracle.params(getattr(A, f"ALGO_{algorithm}"), check_every=101, termination_reltol=0.0)
    prm.sufficient_decay = prm.necessary_decay = 0.0
    prm.artificial_decay = 2.0
    st, _ = _state(handle, lp, prm)
    got = st.solve_blocks(1).err
    e = st.kkt(A.VEC_SOL)  # evaluated anew, by the tile engine
    for f in ("primal", "dual", "gap", "primal_scale", "dual_scale", "gap_scale"):
        a, b = getattr(got, f), getattr(e, f)
        assert abs(a - b) <= 1e-9 * max(1.0, abs(b)), f


@pytest.mark.parametrize("name,ctas", [("31x62x4", 1), ("100x900x4", 4), ("1000x2000x5", 8)])
@pytest.mark.parametrize("check_every,steps", [(101, 250), (257, 300)])
def test_blocks_fp32(handle, name, ctas, check_every, steps):
    from coolpdlp import native, _abi as A
    lp = _lp(name)
    prm = A.default_params_py(A.ALGO_PDLP)
    prm.float_type = A.VAL_F32
    prm.check_every = check_every
    tiles = native.copy_params(prm)
    tiles.tile_nnz = 128
    st, lay = _state(handle, lp, prm)
    assert (lay["engine"], lay["resident_ctas"]) == ("resident", ctas)
    ref, lay = _state(handle, lp, tiles)
    assert lay["engine"] == "tiles"
    st.step(steps)
    ref.step(steps)
    for which in (A.VEC_SOL, A.VEC_SOL_AVG):
        for a, b in zip(st.vectors(which), ref.vectors(which)):
            assert np.linalg.norm(a - b) <= 4e-5 * max(1.0, np.linalg.norm(b))


@pytest.mark.parametrize("name", ["31x62x4", "62x400x5", "100x500x6", "255x513x6"])
def test_power_method_over_several_launches(handle, name):
    from coolpdlp import native, _abi as A
    lp = _lp(name)
    prm = A.default_params_py(A.ALGO_PDLP)
    prm.power_tol_override = 1e-300
    P = native.Problem(handle, _struct(lp), prm)
    assert P.layout()["A"]["engine"] == "resident"
    d1, d2 = P.scaling()
    scaled = d1[:, None] * lp.to_scipy().toarray() * d2[None, :]
    want = np.linalg.norm(scaled, 2)
    for limit in (1023, 1024, 3000):
        prm.power_maxiter_override = limit
        norm, its = P.spectral_norm(prm)
        assert its == limit + 1
    assert abs(norm - want) <= 1e-9 * want


def test_batch_on_two_ctas(handle, oracle):
    """An FP32 LP below the cluster sizes whose 9,000 columns outgrow one CTA's
    shared memory: two CTAs, alone and in a batch."""
    from coolpdlp import generators as G, native, _abi as A
    rng = np.random.RandomState(11)
    m, n, nnz = 64, 9000, 2900
    cols = np.arange(nnz)
    rows = cols % m
    vals = 1.0 + rng.rand(nnz)
    colptr, rowval, nzval = G.csc_from_triplets(m, n, rows, cols, vals)
    lp = G.LPData(m, n, colptr, rowval, nzval, rng.rand(n) - 0.3, np.zeros(n), np.full(n, 10.0),
                  np.full(m, -np.inf), 20.0 + rng.rand(m))
    prm = A.default_params_py(A.ALGO_PDLP)
    prm.float_type = A.VAL_F32
    _, lay = _state(handle, lp, prm)
    assert (lay["engine"], lay["resident_ctas"]) == ("resident", 2)
    xo, _, so = oracle.solve(lp, oracle.params())
    xs, _, st = native.batch_solve(handle, [_struct(lp)] * 3, prm)
    assert so["termination_status"] == 0 and [s.termination_status for s in st] == [0] * 3
    assert np.array_equal(xs[0], xs[1]) and np.array_equal(xs[0], xs[2])
    oo = float(lp.c @ xo)
    assert abs(float(lp.c @ xs[0]) - oo) <= 1e-2 * max(1.0, abs(oo))
