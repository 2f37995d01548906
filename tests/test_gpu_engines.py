"""Which engine a problem's steps run on (cpdlp_problem_engine), where the choice
follows from the LP's sizes and row lengths alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _layout(handle, lp, **fields):
    from coolpdlp import native, _abi as A
    prm = A.default_params_py(A.ALGO_PDLP)
    for k, v in fields.items():
        setattr(prm, k, v)
    S = native.LPStruct(lp.m, lp.n, lp.colptr, lp.rowval, lp.nzval, lp.c, lp.lv, lp.uv, lp.lc, lp.uc)
    lay = native.Problem(handle, S, prm).layout()
    assert lay["A"]["resident_ctas"] == lay["At"]["resident_ctas"]
    return lay["A"]["engine"], lay["At"]["engine"], lay["A"]["resident_ctas"]


@pytest.mark.parametrize("name,float_type,want", [
    ("200x400x5", "F64", ("resident", "resident", 4)), ("100x200x5", "F64", ("resident", "resident", 1)),
    ("200x400x5", "F32", ("resident", "resident", 1)), ("1000x2000x5", "F32", ("resident", "resident", 8)),
    ("20000x40000x5", "F64", ("slices", "slices", 0)), ("20000x40000x5", "F32", ("slices", "slices", 0))])
def test_engine_by_size(handle, name, float_type, want):
    from coolpdlp import generators as G, _abi as A
    m, n, k = (int(v) for v in name.split("x"))
    assert _layout(handle, G.random_sparse_lp(m, n, k, seed=1), float_type=getattr(A, f"VAL_{float_type}")) == want


def test_engine_by_request(handle):
    from coolpdlp import generators as G, _abi as A
    lp = G.random_sparse_lp(1000, 2000, 5, seed=1)
    assert _layout(handle, lp, matrix_type=A.FMT_ELL) == ("ell", "ell", 0)
    assert _layout(handle, lp, tile_nnz=128) == ("tiles", "tiles", 0)


def _even_rows(m, per_row):
    """m x m with `per_row` entries in every row and every column."""
    from coolpdlp import generators as G
    rng = np.random.RandomState(m + per_row)
    shifts = np.append(0, 1 + rng.choice(m - 1, per_row - 1, False))
    cols = (np.arange(m)[:, None] + shifts[None, :]) % m
    rows = np.repeat(np.arange(m), per_row)
    colptr, rowval, nzval = G.csc_from_triplets(m, m, rows, cols.ravel(), rng.randn(rows.size))
    return G.LPData(m, m, colptr, rowval, nzval, rng.rand(m), np.zeros(m), np.full(m, 10.0),
                    np.full(m, -np.inf), np.full(m, 5.0))


@pytest.mark.parametrize("m,per_row,narrow,want", [
    (5000, 32, False, "slices"), (5000, 33, False, "tiles"), (15999, 64, False, "tiles"),
    (16000, 64, False, "slices"), (2000, 24, True, "slices"), (2000, 25, True, "tiles"),
    (15999, 33, True, "tiles"), (16000, 33, True, "slices")])
def test_fp32_rows_of_many_entries(handle, m, per_row, narrow, want):
    """Slices need many rows where a row has many entries (FP32): the edges of
    the rule."""
    from coolpdlp import _abi as A
    lp = _even_rows(m, per_row)
    if narrow:
        lp.nzval = np.sign(lp.nzval)
    assert _layout(handle, lp, float_type=A.VAL_F32) == (want, want, 0)


@pytest.mark.parametrize("m,per_row,want", [(40000, 55, "slices"), (22000, 100, "ell"), (10500, 200, "slices")])
def test_fp64_of_large_lps_by_row_length(handle, m, per_row, want):
    """From 2^21 nonzeros FP64 engines follow the row lengths, not a timing run
    (their roundings differ): the iterates are those of the tiles to rounding."""
    from coolpdlp import native, _abi as A
    lp = _even_rows(m, per_row)
    assert lp.nzval.size >= 1 << 21
    assert _layout(handle, lp) == (want, want, 0)
    S = native.LPStruct(lp.m, lp.n, lp.colptr, lp.rowval, lp.nzval, lp.c, lp.lv, lp.uv, lp.lc, lp.uc)
    got = []
    for tile in (0, 512):
        prm = A.default_params_py(A.ALGO_PDLP)
        prm.power_maxiter_override = 20
        prm.tile_nnz = tile
        if tile:
            prm.matrix_type = A.FMT_CSR
        st = native.State(native.Problem(handle, S, prm), prm)
        st.step(20)
        got.append(st.vectors(A.VEC_SOL))
    for a, b in zip(*got):
        assert np.max(np.abs(a - b)) <= 1e-9 * max(1.0, np.max(np.abs(b)))


def test_power_method_does_not_follow_the_timing(handle):
    """A large LP with +-1 storage steps on ELL or tiles, whichever was faster
    when timed; its |A| is that of the tiles, bit for bit, either way."""
    from coolpdlp import generators as G, native, _abi as A
    lp = G.multicommodity_flow_lp(side=128, K=12, seed=2)
    assert lp.nzval.size >= 1 << 21
    S = native.LPStruct(lp.m, lp.n, lp.colptr, lp.rowval, lp.nzval, lp.c, lp.lv, lp.uv, lp.lc, lp.uc)
    norms = []
    for tile in (0, 512):
        prm = A.default_params_py(A.ALGO_PDLP)
        prm.float_type = A.VAL_F32
        prm.tile_nnz = tile
        if tile:
            prm.matrix_type = A.FMT_CSR
        norms.append(native.Problem(handle, S, prm).spectral_norm(prm))
    assert norms[0] == norms[1]


@pytest.mark.parametrize("narrow", [False, True])
def test_fp32_slices_of_wide_rows_are_the_tile_engines_bits(handle, narrow):
    """16,400 rows of 0 to 64 entries (and a few of 65 and 300) and as many columns
    of about 30 on slices: the iterates have the tile engine's bits."""
    from coolpdlp import generators as G, native, _abi as A
    rng = np.random.RandomState(12)
    m = 16400
    lengths = np.arange(m) % 65
    lengths[:40], lengths[40:44] = 65, 300
    rows = np.repeat(np.arange(m), lengths)
    cols = np.concatenate([(i * 97 + np.sort(rng.choice(m, k, False))) % m for i, k in enumerate(lengths)])
    vals = rng.randn(rows.size)
    colptr, rowval, nzval = G.csc_from_triplets(m, m, rows, cols, np.sign(vals) if narrow else vals)
    lp = G.LPData(m, m, colptr, rowval, nzval, rng.rand(m), np.zeros(m), np.full(m, 10.0),
                  np.full(m, -np.inf), np.full(m, 5.0))
    S = native.LPStruct(lp.m, lp.n, lp.colptr, lp.rowval, lp.nzval, lp.c, lp.lv, lp.uv, lp.lc, lp.uc)
    prm = A.default_params_py(A.ALGO_PDLP)
    prm.float_type = A.VAL_F32
    got = []
    for tile in (0, 256):
        prm.tile_nnz = tile
        P = native.Problem(handle, S, prm)
        lay = P.layout()
        assert lay["A"]["engine"] == lay["At"]["engine"] == ("tiles" if tile else "slices")
        assert lay["A"]["tile_nnz"] == lay["At"]["tile_nnz"] == 256
        st = native.State(P, prm, np.linspace(0, 1, m), np.linspace(-1, 1, m))
        st.step(30)
        got.append([v for which in (A.VEC_SOL, A.VEC_SOL_AVG) for v in st.vectors(which)])
    for a, b in zip(*got):
        assert np.array_equal(a, b)
