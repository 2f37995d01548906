"""The solver's measured workloads.

Each case is one thing a program does with this library, through its public
entry points: `mul!` of a pluggable sparse matrix, a whole `solve`, a stretch of
`solve!` on a resident problem, a batch of LPs in one call.  The matrices are
the three families the package names (random sparse, power-law rows, grid
multicommodity flow); they are drawn on the GPU from the seed.

listed() gives the fixed cases, draw(rng) more of the same ranges, prepare()
what a program holds before the call, run() the call, work() the bytes and
operations it cannot do without, and exact() its result in plain FP64 torch.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "coolpdlp.jl_gb300"))

import coolpdlp as cp  # noqa: E402
from coolpdlp import _abi, native  # noqa: E402

DEV = "cuda"
MATRIX = {"csr": cp.GPUSparseMatrixCSR, "ell": cp.GPUSparseMatrixELL, "coo": cp.GPUSparseMatrixCOO}


def listed():
    return [
        # mul! of a small LP's matrix: one product of a few microseconds, where
        # the launch and the call itself are what a program waits for
        {"name": "mul_csr_f64_small", "kind": "mul", "format": "csr", "dtype": "f64",
         "family": "random", "m": 1000, "n": 2000, "per_col": 5, "beta": 0.0},
        # the same for the triplet format, odd sizes, accumulating (beta != 0)
        {"name": "mul_coo_f64_odd", "kind": "mul", "format": "coo", "dtype": "f64",
         "family": "random", "m": 50021, "n": 99877, "per_col": 5, "beta": 0.5},
        # ELL on its natural matrix: grid flow incidence, 3 entries a column
        {"name": "mul_ell_f32_flow", "kind": "mul", "format": "ell", "dtype": "f32",
         "family": "flow", "side": 128, "K": 8, "beta": 0.0},
        # a large irregular CSR product
        {"name": "mul_csr_f32_powerlaw", "kind": "mul", "format": "csr", "dtype": "f32",
         "family": "powerlaw", "m": 1000000, "n": 2000000, "nnz": 12000000, "beta": 0.0},
        # a whole solve of the 1,000 x 2,000 random LP to 1e-4 (Float64)
        {"name": "solve_f64_random", "kind": "solve", "dtype": "f64", "algorithm": "PDLP",
         "family": "random", "m": 1000, "n": 2000, "per_col": 5, "reltol": 1e-4, "passes": 10000},
        # a served-size flow LP, PDHG, ended by its pass limit
        {"name": "solve_f64_flow_pdhg", "kind": "solve", "dtype": "f64", "algorithm": "PDHG",
         "family": "flow", "side": 33, "K": 5, "reltol": 1e-8, "passes": 2000},
        # a large LP end to end: upload, scaling, step size, 1,000 iterations, download
        {"name": "solve_f32_powerlaw", "kind": "solve", "dtype": "f32", "algorithm": "PDLP",
         "family": "powerlaw", "m": 400000, "n": 800000, "nnz": 4800000, "reltol": 1e-6,
         "passes": 1000},
        # the large power-law LP resident on the GPU: solve! blocks (100
        # iterations and a check each), then the solution
        {"name": "blocks_f32_powerlaw", "kind": "blocks", "dtype": "f32", "algorithm": "PDLP",
         "family": "powerlaw", "m": 2000000, "n": 4000000, "nnz": 24000000, "blocks": 3},
        # the same in Float64, a quarter of the size
        {"name": "blocks_f64_powerlaw", "kind": "blocks", "dtype": "f64", "algorithm": "PDLP",
         "family": "powerlaw", "m": 500000, "n": 1000000, "nnz": 6000000, "blocks": 3},
        # the 256 x 256 grid, 16 commodity flow LP (+-1 storage)
        {"name": "blocks_f32_flow", "kind": "blocks", "dtype": "f32", "algorithm": "PDLP",
         "family": "flow", "side": 256, "K": 16, "blocks": 3},
        # many random LPs of uneven size in one call, FP32 iterates
        {"name": "batch_f32", "kind": "batch", "dtype": "f32", "count": 256, "m_lo": 50,
         "m_hi": 2000, "reltol": 1e-4, "passes": 8000},
        # and in Float64, smaller LPs
        {"name": "batch_f64", "kind": "batch", "dtype": "f64", "count": 128, "m_lo": 50,
         "m_hi": 600, "reltol": 1e-4, "passes": 8000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mul", "mul", "solve", "blocks", "blocks", "batch"])
    dtype = rng.choice(["f32", "f64"])
    family = rng.choice(["random", "powerlaw", "flow"])
    if family == "random":
        m = _log_int(rng, 100, 20000 if kind == "solve" else 1000000)
        fam = {"m": m, "n": 2 * m + rng.randint(-m // 4, m // 4), "per_col": rng.randint(3, 8)}
    elif family == "powerlaw":
        m = _log_int(rng, 2000, 400000 if kind == "solve" else 1500000)
        fam = {"m": m, "n": 2 * m + rng.randint(-m // 4, m // 4), "nnz": 12 * m}
    else:
        fam = {"side": _log_int(rng, 8, 64 if kind == "solve" else 256), "K": rng.randint(2, 16)}
    if kind == "mul":
        formats = ["csr", "coo"] if family == "powerlaw" else ["csr", "ell", "coo"]
        return {"kind": kind, "format": rng.choice(formats), "dtype": dtype, "family": family,
                "beta": rng.choice([0.0, 0.5]), **fam}
    if kind == "solve":
        return {"kind": kind, "dtype": dtype, "algorithm": rng.choice(["PDLP", "PDHG"]),
                "family": family, "reltol": 1e-8, "passes": 100 * rng.randint(3, 10), **fam}
    if kind == "blocks":
        return {"kind": kind, "dtype": dtype, "algorithm": rng.choice(["PDLP", "PDLP", "PDHG"]),
                "family": family, "blocks": rng.randint(1, 3), **fam}
    return {"kind": kind, "dtype": dtype, "count": _log_int(rng, 16, 200), "m_lo": 50,
            "m_hi": _log_int(rng, 300, 600 if dtype == "f64" else 2000), "reltol": 1e-4,
            "passes": 8000}


# ---------------------------------------------------------------------------
# the LP families, drawn from a seed (device random numbers; every sum that
# enters an input is a host sum in a fixed order)
# ---------------------------------------------------------------------------
class LP:
    """min c'x, lv <= x <= uv, lc <= Ax <= uc; A in 1-based CSC."""

    def __init__(self, m, n, rows, cols, vals, c, lv, uv, lc, uc):
        self.m, self.n, self.nnz = m, n, int(vals.size)
        self.rows, self.cols = rows, cols  # 0-based, column by column
        counts = np.bincount(cols, minlength=n)
        self.colptr = np.concatenate([[1], 1 + np.cumsum(counts)]).astype(np.int64)
        self.rowval, self.nzval = rows + 1, vals
        self.c, self.lv, self.uv, self.lc, self.uc = c, lv, uv, lc, uc


def _uniform(g, count, lo=0.0, hi=1.0):
    u = torch.rand(count, generator=g, device=DEV, dtype=torch.float64)
    return (lo + (hi - lo) * u).cpu().numpy()


def _normal(g, count):
    return torch.randn(count, generator=g, device=DEV, dtype=torch.float64).cpu().numpy()


def _entries(m, keys):
    """(rows, cols) of the distinct entries col * m + row, column by column."""
    keys = torch.unique(keys)
    return (keys % m).cpu().numpy(), torch.div(keys, m, rounding_mode="floor").cpu().numpy()


def _planted(g, m, n, rows, cols, vals):
    """Feasible and bounded by construction: x* in [0, 10] with some entries at
    0, half of the rows equalities at A x*, the others <= with slack, and
    c = A'y* + s for multipliers y* of the right signs."""
    xs = _uniform(g, n, 0.0, 10.0)
    low = _uniform(g, n) < 0.3
    xs[low] = 0.0
    s = np.where(low, _uniform(g, n), 0.0)
    ax = np.bincount(rows, weights=vals * xs[cols], minlength=m)
    n_eq = m // 2
    lc = np.full(m, -np.inf)
    lc[:n_eq] = ax[:n_eq]
    uc = ax + _uniform(g, m)
    uc[:n_eq] = ax[:n_eq]
    ys = _normal(g, m)
    ys[n_eq:] = -np.abs(ys[n_eq:])
    c = np.bincount(cols, weights=vals * ys[rows], minlength=n) + s
    return LP(m, n, rows, cols, vals, c, np.zeros(n), np.full(n, 10.0), lc, uc)


def _random_lp(g, m, n, per_col):
    k = min(per_col, m)
    rows = torch.randint(0, m, (n, k), generator=g, device=DEV)
    keys = torch.arange(n, device=DEV)[:, None] * m + rows
    rows, cols = _entries(m, keys.reshape(-1))
    return _planted(g, m, n, rows, cols, _normal(g, rows.size))


def _powerlaw_lp(g, m, n, nnz):
    """Row lengths Pareto with tail exponent 1.5 (capped at 20,000 and n / 2),
    columns uniform, values N(0,1) times a row factor in [1e-3, 1e3]."""
    u = torch.rand(m, generator=g, device=DEV, dtype=torch.float64)
    length = torch.ceil(nnz / (3.0 * m) * (1.0 - u) ** (-1.0 / 1.5))
    length = length.clamp(max=min(20000, n // 2)).long()
    row = torch.repeat_interleave(torch.arange(m, device=DEV), length)
    col = torch.randint(0, n, row.shape, generator=g, device=DEV)
    rows, cols = _entries(m, col * m + row)
    factor = np.exp(_uniform(g, m, math.log(1e-3), math.log(1e3)))
    return _planted(g, m, n, rows, cols, _normal(g, rows.size) * factor[rows])


def _flow_lp(g, side, K):
    """K-commodity min-cost flow on a directed side x side grid: conservation
    rows per node and commodity (equalities), a capacity row per arc, +-1
    entries; capacities are raised where an L-shaped routing needs them."""
    nodes = side * side
    idx = np.arange(nodes).reshape(side, side)
    rt, rh, dt, dh = (a.ravel() for a in (idx[:, :-1], idx[:, 1:], idx[:-1], idx[1:]))
    tail, head = np.concatenate([rt, rh, dt, dh]), np.concatenate([rh, rt, dh, dt])
    arcs, h, v = tail.size, rt.size, dt.size
    ends = (_uniform(g, 2 * K) * nodes).astype(np.int64)
    src, dst = ends[:K], ends[K:]
    dst = np.where(src == dst, (dst + 1) % nodes, dst)
    demand, cost = _uniform(g, K, 1.0, 10.0), _uniform(g, arcs, 1.0, 10.0)
    cap, load = _uniform(g, arcs, 5.0, 40.0), np.zeros(arcs)
    for k in range(K):  # along the source's row, then along the target's column
        (r0, c0), (r1, c1) = divmod(int(src[k]), side), divmod(int(dst[k]), side)
        a, b = min(c0, c1), max(c0, c1)
        load[(0 if c1 > c0 else h) + r0 * (side - 1) + np.arange(a, b)] += demand[k]
        a, b = min(r0, r1), max(r0, r1)
        load[2 * h + (0 if r1 > r0 else v) + np.arange(a, b) * side + c1] += demand[k]
    n, m = arcs * K, nodes * K + arcs
    var = np.arange(n)
    arc, com = var // K, var % K
    rows = np.stack([tail[arc] * K + com, head[arc] * K + com, nodes * K + arc], axis=1)
    vals = np.tile([1.0, -1.0, 1.0], (n, 1))
    swap = rows[:, 0] > rows[:, 1]  # rows ascending inside each column
    rows[swap, :2], vals[swap, :2] = rows[swap, 1::-1], vals[swap, 1::-1]
    b = np.zeros(nodes * K)
    np.add.at(b, src * K + np.arange(K), demand)
    np.add.at(b, dst * K + np.arange(K), -demand)
    return LP(m, n, rows.ravel(), np.repeat(var, 3), vals.ravel(), cost[arc], np.zeros(n),
              np.full(n, np.inf), np.concatenate([b, np.full(arcs, -np.inf)]),
              np.concatenate([b, np.maximum(cap, load)]))


def _family(case, g):
    if case["family"] == "random":
        return _random_lp(g, case["m"], case["n"], case["per_col"])
    if case["family"] == "powerlaw":
        return _powerlaw_lp(g, case["m"], case["n"], case["nnz"])
    return _flow_lp(g, case["side"], case["K"])


def _batch(case, g):
    """Random LPs, m log-uniform, n = 2m, 3 to 8 nonzeros a column."""
    count = case["count"]
    sizes = np.random.RandomState(count)  # the same sizes from any seed
    u, per = sizes.rand(count), sizes.randint(3, 9, count)
    ms = np.round(case["m_lo"] * (case["m_hi"] / case["m_lo"]) ** u).astype(int)
    return [_random_lp(g, int(m), 2 * int(m), int(k)) for m, k in zip(ms, per)]


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _algorithm(case):
    T = np.float32 if case["dtype"] == "f32" else np.float64
    return cp.Algorithm(case.get("algorithm", "PDLP"), T,
                        termination_reltol=case.get("reltol", 0.0),
                        max_kkt_passes=case.get("passes", 10**9), time_limit=1e6)


def _struct(lp):
    return native.LPStruct(lp.m, lp.n, lp.colptr, lp.rowval, lp.nzval, lp.c, lp.lv, lp.uv, lp.lc,
                           lp.uc)


def prepare(case, seed):
    g = _generator(seed)
    if case["kind"] == "batch":
        return {"kind": "batch", "handle": native.default_handle(),
                "lps": [_struct(lp) for lp in _batch(case, g)], "algo": _algorithm(case)}
    lp = _family(case, g)
    if case["kind"] == "mul":
        T = torch.float32 if case["dtype"] == "f32" else torch.float64
        A = MATRIX[case["format"]](cp.CSCMatrix(lp.m, lp.n, lp.colptr, lp.rowval, lp.nzval),
                                   np.float32 if case["dtype"] == "f32" else np.float64)
        b, c = (torch.randn(k, generator=g, device=DEV, dtype=T) for k in (lp.n, lp.m))
        return {"kind": "mul", "A": A, "b": b, "c": c, "alpha": 1.0, "beta": case["beta"]}
    algo = _algorithm(case)
    if case["kind"] == "solve":
        milp = cp.MILP(c=lp.c, lv=lp.lv, uv=lp.uv, lc=lp.lc, uc=lp.uc,
                       A=cp.CSCMatrix(lp.m, lp.n, lp.colptr, lp.rowval, lp.nzval))
        return {"kind": "solve", "milp": milp, "algo": algo}
    problem = native.Problem(native.default_handle(), _struct(lp), algo.params)
    return {"kind": "blocks", "problem": problem, "state": native.State(problem, algo.params),
            "blocks": case["blocks"], "dtype": case["dtype"]}


def _eltype(v, algo_T):
    """The solution in the iterates' type, as the reference returns it."""
    return torch.from_numpy(v).to(torch.float32 if algo_T in (np.float32, "f32") else torch.float64)


def _outputs(x, y, T, err, omega, passes, status):
    return {"x": _eltype(x, T), "y": _eltype(y, T), "passes": int(passes), "status": int(status),
            "omega": float(omega),
            "err": [float(e) for e in (err.primal, err.primal_scale, err.dual, err.dual_scale,
                                       err.gap, err.gap_scale)]}


def run(state):
    if state["kind"] == "mul":
        return state["A"].mul(state["c"], state["b"], state["alpha"], state["beta"])
    if state["kind"] == "solve":
        sol, st = cp.solve(state["milp"], state["algo"])
        return _outputs(sol.x, sol.y, state["algo"].T, st.err, st.omega, st.kkt_passes,
                        st.termination_status)
    if state["kind"] == "blocks":
        st = state["state"].solve_blocks(state["blocks"])
        x, y = state["state"].solution()
        return _outputs(x, y, state["dtype"], st.err, st.omega, st.kkt_passes,
                        st.termination_status)
    xs, ys, sts = native.batch_solve(state["handle"], state["lps"], state["algo"].params)
    T = state["algo"].T
    return {"x": _eltype(np.concatenate(xs), T), "y": _eltype(np.concatenate(ys), T),
            "passes": np.array([s.kkt_passes for s in sts]),
            "status": np.array([s.termination_status for s in sts])}


# ---------------------------------------------------------------------------
def _sizes(case):
    """(m, n, nnz) expected of the case's LP."""
    if case["family"] == "random":
        return case["m"], case["n"], case["n"] * min(case["per_col"], case["m"])
    if case["family"] == "powerlaw":
        return case["m"], case["n"], case["nnz"]
    arcs = 4 * case["side"] * (case["side"] - 1)
    return case["side"] ** 2 * case["K"] + arcs, arcs * case["K"], 3 * arcs * case["K"]


def work(case):
    """mul!: the matrix in its format and the vectors.  Iterations: both
    matrices (no values for +-1 entries in FP32) and the step's vectors once per
    iteration where the LP exceeds the on-chip memory (100 MB), once in all
    where it does not; a solve also reads the caller's arrays once.  A solve to
    a tolerance is counted at 1,000 iterations (a batch: each LP)."""
    s = 4 if case["dtype"] == "f32" else 8
    if case["kind"] == "batch":
        mean = (case["m_hi"] - case["m_lo"]) / math.log(case["m_hi"] / case["m_lo"])
        m, n, nnz = (int(case["count"] * v) for v in (mean, 2 * mean, 11 * mean))
    else:
        m, n, nnz = _sizes(case)
    if case["kind"] == "mul":
        per = {"csr": 4, "ell": 4, "coo": 8}[case["format"]] + s
        rows = 4 * m if case["format"] == "csr" else 0
        return {"bytes": per * nnz + rows + s * (n + m * (2 if case["beta"] else 1)),
                "flops": 2 * nnz}
    v = 0 if case.get("family") == "flow" and case["dtype"] == "f32" else s
    avg = case.get("algorithm", "PDLP") == "PDLP"
    step = 2 * nnz * (v + 4) + 4 * (m + n) + s * ((9 if avg else 7) * n + (7 if avg else 5) * m)
    iters = (100 * case["blocks"] if case["kind"] == "blocks" else
             case["passes"] if case["kind"] == "solve" and case["passes"] <= 2000 else 1000)
    host = 0 if case["kind"] == "blocks" else 16 * nnz + 32 * n + 24 * m
    return {"bytes": step * (iters if step > 100e6 else 1) + host + 8 * (m + n),
            "flops": iters * (4 * nnz + 20 * (m + n))}


# ---------------------------------------------------------------------------
# exact(): the same computation in FP64 torch
# ---------------------------------------------------------------------------
def _splitmix(seed, counters):
    with np.errstate(over="ignore"):
        z = np.uint64(seed) + (counters + np.uint64(1)) * np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))


def _start_vector(seed, n):
    """The power method's Gaussian start vector (SplitMix64, Box-Muller)."""
    i = 2 * np.arange(n, dtype=np.uint64)
    u1, u2 = (((_splitmix(seed, k) >> np.uint64(11)) + np.uint64(1)).astype(np.float64) / 2.0**53
              for k in (i, i + np.uint64(1)))
    return torch.from_numpy(np.sqrt(-2.0 * np.log(u1)) * np.cos(2.0 * math.pi * u2)).to(DEV)


class _Exact:
    """PDLP / PDHG on one LP, restated in FP64."""

    def __init__(self, lp, case):
        p = _algorithm(case).params
        self.p, self.pdlp, self.f32 = p, p.algorithm == _abi.ALGO_PDLP, case["dtype"] == "f32"
        t = lambda v: torch.from_numpy(np.ascontiguousarray(v)).to(DEV)  # noqa: E731
        m, n = lp.m, lp.n
        rows, cols, vals = t(lp.rows), t(lp.cols), t(lp.nzval)
        order = torch.argsort(rows * n + cols)
        ptr = lambda k, size: torch.cat([torch.zeros(1, dtype=torch.long, device=DEV),  # noqa: E731
                                         torch.cumsum(torch.bincount(k, minlength=size), 0)])
        d1, d2 = torch.ones(m, device=DEV).double(), torch.ones(n, device=DEV).double()
        inv_sqrt = lambda v: torch.where(v == 0, 1.0, 1.0 / torch.sqrt(v))  # noqa: E731
        norm = lambda k, size, a, how: torch.zeros(size, device=DEV).double().scatter_reduce_(  # noqa: E731
            0, k, a, how)
        for _ in range(p.ruiz_iter):
            w = (d1[rows] * vals * d2[cols]).abs()
            s1, s2 = norm(rows, m, w, "amax"), norm(cols, n, w, "amax")
            d1, d2 = d1 * inv_sqrt(s1), d2 * inv_sqrt(s2)
        w = (d1[rows] * vals * d2[cols]).abs()
        al = p.chambolle_pock_alpha
        s1, s2 = norm(rows, m, w ** (2 - al), "sum"), norm(cols, n, w**al, "sum")
        if al != 1.0:
            s1, s2 = s1 ** (1 / (2 - al)), s2 ** (1 / al)
        self.d1, self.d2 = d1 * inv_sqrt(s1), d2 * inv_sqrt(s2)
        v = self.d1[rows] * vals * self.d2[cols]
        self.A = torch.sparse_csr_tensor(ptr(rows, m), cols[order], v[order], (m, n))
        self.At = torch.sparse_csr_tensor(ptr(cols, n), rows, v, (n, m))
        self.c, self.lv, self.uv = t(lp.c) * self.d2, t(lp.lv) / self.d2, t(lp.uv) / self.d2
        self.lc, self.uc = t(lp.lc) * self.d1, t(lp.uc) * self.d1
        self.m, self.n = m, n
        fin = lambda b: torch.where(torch.isinf(b), 0.0, b.abs())  # noqa: E731
        comb = torch.maximum(fin(self.lc), fin(self.uc))
        self.scale = (1 + float((comb / self.d1).norm()), 1 + float((self.c / self.d2).norm()))
        cn, bn = float(self.c.norm()), float(comb.norm())
        self.omega = cn / bn if self.pdlp and min(cn, bn) > p.zero_tol else 1.0
        self.eta = p.invnorm_scaling / math.sqrt(self._power())

    def _power(self):
        n3 = (self.n**3 + 2**63) % 2**64 - 2**63
        tol, x, it = 2.220446049250313e-16 * n3, _start_vector(int(self.p.power_seed), self.n), 0
        while True:
            ax = self.At @ (self.A @ x)
            theta = float(x @ ax)
            res = float((ax - theta * x).norm())
            x = ax / ax.norm()
            it += 1
            if it > self.n or res <= tol or (self.f32 and res <= 1e-2 * theta):
                return theta

    def _err(self, x, y):
        s, g = self.A @ x, self.c - self.At @ y
        lmin, umax = torch.isinf(self.lv), torch.isinf(self.uv)
        r = torch.where(lmin, torch.where(umax, 0.0, g.clamp(max=0)),
                        torch.where(umax, g.clamp(min=0), g))
        safe = lambda b, q: torch.where(torch.isinf(b), q, b * q)  # noqa: E731
        dual = lambda lo, up, z: float((safe(up, (-z).clamp(min=0))  # noqa: E731
                                        - safe(lo, (-(-z).clamp(max=0)))).sum())
        pc, pv = dual(self.lc, self.uc, y), dual(self.lv, self.uv, r)
        cx = float(self.c @ x)
        box = torch.minimum(self.uc, torch.maximum(self.lc, s))
        return (float(((s - box) / self.d1).norm()), self.scale[0],
                float(((g - r) / self.d2).norm()), self.scale[1],
                abs(cx + pc + pv), 1 + abs(pc + pv) + abs(cx))

    @staticmethod
    def _rel(e):
        return max(e[0] / e[1], e[2] / e[3], e[4] / e[5])

    def _abs(self, e):
        w = self.omega
        return math.sqrt(w * w * e[0] ** 2 + e[2] ** 2 / (w * w) + e[4] ** 2)

    def run(self, max_blocks, reltol, max_passes):
        p = self.p
        x, y = torch.zeros(self.n, device=DEV).double(), torch.zeros(self.m, device=DEV).double()
        xa, ya, xr, yr = x, y, x, y
        er, passes, inner, total, es = None, 0, 0, 0, 0.0
        for _ in range(max_blocks):
            tau, sig = self.eta / self.omega, self.eta * self.omega
            for _ in range(p.check_every):
                xl, yl, xal, yal = x, y, xa, ya
                x = torch.minimum(self.uv, torch.maximum(self.lv, x - tau * (self.c - self.At @ y)))
                s = self.A @ (2 * x - xl)
                box = torch.minimum(-self.lc, torch.maximum(-self.uc, y / sig - s))
                y = y - sig * s - sig * box
                if self.pdlp:
                    a, b = self.eta / (self.eta + es), es / (self.eta + es)
                    xa, ya, es = a * x + b * xa, a * y + b * ya, es + self.eta
            passes += p.check_every
            err = self._err(x, y)
            status = (0 if self._rel(err) <= reltol else 2 if passes >= max_passes else 3)
            if status != 3:
                break
            if not self.pdlp:
                continue
            inner, total = inner + p.check_every, total + p.check_every
            ea, el, eal = self._err(xa, ya), self._err(xl, yl), self._err(xal, yal)
            from_avg = not self._abs(err) < self._abs(ea)
            cand = ea if from_avg else err
            last = min(self._abs(el), self._abs(eal))
            er = er or self._err(xr, yr)
            ac, ar = self._abs(cand), self._abs(er)
            if (ac <= p.sufficient_decay * ar or (ac <= p.necessary_decay * ar and ac > last)
                    or inner >= p.artificial_decay * total):
                if from_avg:
                    x, y = xa, ya
                dx, dy = float((x - xr).norm()), float((y - yr).norm())
                if min(dx, dy) > p.zero_tol:
                    th = p.primal_weight_damping
                    self.omega = math.exp(th * math.log(dy / dx) + (1 - th) * math.log(self.omega))
                xa, ya, xr, yr = torch.zeros_like(x), torch.zeros_like(y), x, y
                er, es, inner = cand, 0.0, 0
        return {"x": self.d2 * x, "y": self.d1 * y, "passes": None, "status": None,
                "omega": torch.tensor(self.omega, dtype=torch.float64),
                "err": [torch.tensor(e, dtype=torch.float64) for e in err]}


def exact(case, seed):
    if case["kind"] == "batch":
        return None  # hundreds of solves, one after the other: minutes
    g = _generator(seed)
    lp = _family(case, g)
    if case["kind"] == "mul":
        T = torch.float32 if case["dtype"] == "f32" else torch.float64
        b, c = (torch.randn(k, generator=g, device=DEV, dtype=T).double() for k in (lp.n, lp.m))
        vals = torch.from_numpy(lp.nzval).to(DEV).to(T).double()  # the matrix as it is stored
        rows, cols = torch.from_numpy(lp.rows).to(DEV), torch.from_numpy(lp.cols).to(DEV)
        s = torch.zeros(lp.m, device=DEV).double().index_add_(0, rows, vals * b[cols])
        return s + case["beta"] * c if case["beta"] else s
    E = _Exact(lp, case)
    if case["kind"] == "blocks":
        return E.run(case["blocks"], 0.0, 10**9)
    return E.run(10**6, case["reltol"], case["passes"])
