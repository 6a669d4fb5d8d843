"""The work that programs give this library, as cases to time: interior-point
and trajectory-optimisation KKT systems and SPD grid operators, factored,
solved and refined through ``smfg.Solver``, ``batch.BatchSolver`` and
``ipm.IpmSession``.

A case names a matrix family with its sizes and what one pass does with it:

  step    factor new values and solve (the inner step of every caller)
  refine  factor, solve and refine to omega <= 1e-12 (a caller that needs full
          backward accuracy; the only way a mixed-precision factor is used)
  solve   solve with the factor kept from before (several right-hand sides of
          one matrix, the corrector solves of an interior-point iteration)

The analysis of a pattern is made once per process and kept, as every caller
keeps it over its refactorizations; each state has a plan of its own, and new
values and right-hand sides from its seed.
"""
import functools
import math

import numpy as np
import torch

from opt_solver_b200 import batch, ipm, smfg

DEV = "cuda"
NX, NU = 12, 4  # a trajectory stage: states and controls
OMEGA = 1e-12


def listed():
    return [
        # A model-predictive controller's system, ten stages, in host memory:
        # the smallest call, where latency and launches are everything.
        {"name": "traj_10_host", "kind": "traj", "T": 10, "nrhs": 1, "do": "step", "host": True},
        # One long trajectory with the eight right-hand sides of a sensitivity
        # solve: a deep tree of small indefinite fronts.
        {"name": "traj_200_rhs8", "kind": "traj", "T": 200, "nrhs": 8, "do": "step"},
        # A batch of trajectories of uneven horizons, factored as one forest.
        {"name": "batch_256_refine", "kind": "batch", "count": 256, "t_min": 10, "t_max": 200, "nrhs": 8,
         "do": "refine"},
        # The 2D Laplacian of the benchmark: small and medium SPD fronts.
        {"name": "grid2_150", "kind": "grid2", "nx": 150, "ny": 150, "nrhs": 1, "do": "step"},
        # A larger ragged 2D operator, refactored by graph replay.
        {"name": "grid2_701x433_graph", "kind": "grid2", "nx": 701, "ny": 433, "nrhs": 1, "do": "step",
         "graph": True},
        # A small ragged 3D operator in host memory, refined.
        {"name": "grid3_23_host", "kind": "grid3", "nx": 23, "ny": 19, "nz": 21, "nrhs": 3, "do": "refine",
         "host": True},
        # Sixteen right-hand sides against a kept factor of a 40^3 operator.
        {"name": "grid3_40_solve16", "kind": "grid3", "nx": 40, "ny": 40, "nz": 40, "nrhs": 16, "do": "solve"},
        # One right-hand side against a kept factor.
        {"name": "grid3_52_solve1", "kind": "grid3", "nx": 52, "ny": 49, "nz": 50, "nrhs": 1, "do": "solve"},
        # The headline operator, 64^3, in FP64.
        {"name": "grid3_64", "kind": "grid3", "nx": 64, "ny": 64, "nz": 64, "nrhs": 1, "do": "step"},
        # The same in mixed precision, refined to full backward accuracy.
        {"name": "grid3_64_mixed", "kind": "grid3", "nx": 64, "ny": 64, "nz": 64, "nrhs": 1, "do": "refine",
         "mixed": "tf32"},
        # An interior-point iteration's KKT system through a session: host
        # memory, matching scaling, the threshold kernel on every front.
        {"name": "kkt_12_session", "kind": "kkt", "m": 12, "cons": 500, "nrhs": 1, "do": "step", "host": True,
         "session": True, "aptp": False},
        # The benchmark's KKT system in the default (deterministic) mode.
        {"name": "kkt_20_4000", "kind": "kkt", "m": 20, "cons": 4000, "nrhs": 1, "do": "step", "aptp": True},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["traj", "batch", "grid2", "grid3", "grid3", "kkt"])
    nrhs = rng.choice([1, 1, 2, 3, 5, 8, 16])
    if kind == "traj":
        return {"kind": kind, "T": _size(rng, 10, 200), "nrhs": min(nrhs, 8), "do": rng.choice(["step", "refine"]),
                "host": rng.random() < 0.5}
    if kind == "batch":
        return {"kind": kind, "count": _size(rng, 8, 256), "t_min": 10, "t_max": _size(rng, 40, 200),
                "nrhs": min(nrhs, 8), "do": rng.choice(["step", "refine"])}
    if kind == "grid2":
        return {"kind": kind, "nx": _size(rng, 20, 700), "ny": _size(rng, 20, 430), "nrhs": min(nrhs, 8),
                "do": rng.choice(["step", "solve"]), "graph": rng.random() < 0.3}
    if kind == "grid3":
        m = _size(rng, 9, 60)
        dims = {"nx": m, "ny": max(5, int(m * rng.uniform(0.8, 1.05))), "nz": max(5, int(m * rng.uniform(0.8, 1.05)))}
        do = rng.choice(["step", "refine", "solve"])
        if do == "refine":
            nrhs = 1
        case = {"kind": kind, **dims, "nrhs": nrhs, "do": do, "host": rng.random() < 0.3}
        if do == "refine" and rng.random() < 0.6:
            case["mixed"] = rng.choice(["tf32", "bf16"])
        elif do == "step":
            case["graph"] = rng.random() < 0.3
        return case
    m = _size(rng, 6, 18)
    return {"kind": kind, "m": m, "cons": int(m ** 3 * rng.uniform(0.1, 0.45)), "nrhs": min(nrhs, 3),
            "do": rng.choice(["step", "solve"]), "host": rng.random() < 0.5, "aptp": rng.random() < 0.5}


# ---------------------------------------------------------------------------
# Matrices: the pattern of a case, and its values from a seed. Values are made
# in the order of the pattern's triplets and put into CSC order.


class Pattern:
    """Lower CSC (rows ascending in each column) of triplets without
    duplicates; `order` takes values from triplet order to CSC order."""

    def __init__(self, n, rows, cols, **more):
        self.n = int(n)
        lo, hi = np.maximum(rows, cols).astype(np.int64), np.minimum(rows, cols).astype(np.int64)
        order = np.argsort(hi * n + lo, kind="stable")
        self.rows, self.cols = lo[order], hi[order]
        self.ptr = np.zeros(n + 1, np.int32)
        np.cumsum(np.bincount(self.cols, minlength=n), out=self.ptr[1:])
        self.idx = self.rows.astype(np.int32)
        self.order = torch.from_numpy(order).to(DEV)
        self.__dict__.update(more)


def _grid_edges(dims):
    idx = np.arange(int(np.prod(dims))).reshape(dims[::-1])
    a, b = [], []
    for ax in range(idx.ndim):
        n = idx.shape[ax]
        a.append(idx.take(range(1, n), ax).ravel())
        b.append(idx.take(range(n - 1), ax).ravel())
    return np.concatenate(a), np.concatenate(b)


@functools.lru_cache(maxsize=8)
def _grid(dims):
    n = int(np.prod(dims))
    ea, eb = _grid_edges(dims)
    return Pattern(n, np.concatenate([np.arange(n), ea]), np.concatenate([np.arange(n), eb]),
                   ea=torch.from_numpy(ea).to(DEV), eb=torch.from_numpy(eb).to(DEV))


@functools.lru_cache(maxsize=4)
def _kkt(m, cons):
    nh = m ** 3
    ea, eb = _grid_edges((m, m, m))
    rng = np.random.default_rng(m * 100003 + cons)
    j = np.stack([rng.choice(nh, size=4, replace=False) for _ in range(cons)])
    c = nh + np.arange(cons)
    return Pattern(nh + cons, np.concatenate([np.arange(nh), ea, np.repeat(c, 4), c]),
                   np.concatenate([np.arange(nh), eb, j.ravel(), c]), nh=nh, edges=ea.size)


@functools.lru_cache(maxsize=None)
def _traj(T):
    """Stages [x_k, u_k, lambda_{k+1}] for k < T, then x_T."""
    nz, st = NX + NU, 2 * NX + NU
    k = np.arange(T)[:, None] * st
    qi, qj = np.tril_indices(nz)
    ti, tj = np.tril_indices(NX)
    ai, aj = (x.ravel() for x in np.meshgrid(np.arange(NX), np.arange(nz), indexing="ij"))
    d = np.arange(NX)
    rows = [(k + qi), T * st + ti, (k + nz + ai), (k + st + d), (k + nz + d)]
    cols = [(k + qj), T * st + tj, (k + aj), (k + nz + d), (k + nz + d)]
    return Pattern(st * T + NX, np.concatenate([np.ravel(r) for r in rows]),
                   np.concatenate([np.ravel(c) for c in cols]))


def _traj_values(T, gen):
    nz = NX + NU
    f = dict(dtype=torch.float64, device=DEV, generator=gen)
    tril = lambda n: tuple(torch.from_numpy(np.stack(np.tril_indices(n))).to(DEV))  # noqa: E731

    def wishart(count, n):
        g = torch.randn(count, n, 2 * n, **f)
        q = g @ g.transpose(1, 2) + 1e-6 * torch.eye(n, dtype=torch.float64, device=DEV)
        i, j = tril(n)
        return q[:, i, j].reshape(-1)

    ab = torch.cat([torch.eye(NX, dtype=torch.float64, device=DEV) + 0.01 * torch.randn(NX, NX, **f),
                    0.1 * torch.randn(NX, NU, **f)], 1).reshape(-1)
    one = torch.ones(T * NX, dtype=torch.float64, device=DEV)
    return torch.cat([wishart(T, nz), wishart(1, NX), ab.repeat(T), -one, -1e-9 * one])


def _horizons(case):
    rng = np.random.default_rng(case["count"] * 1009 + case["t_max"])
    return [int(t) for t in rng.integers(case["t_min"], case["t_max"] + 1, size=case["count"])]


def _pattern(case):
    if case["kind"] == "traj":
        return _traj(case["T"])
    if case["kind"] == "kkt":
        return _kkt(case["m"], case["cons"])
    return _grid((case["nx"], case["ny"]) + ((case["nz"],) if case["kind"] == "grid3" else ()))


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) & 0x7FFFFFFF)


def _values(case, p, gen):
    """The values of one system on the GPU, CSC order."""
    f = dict(dtype=torch.float64, device=DEV)
    u = lambda n, lo, hi: 10.0 ** (lo + (hi - lo) * torch.rand(n, generator=gen, **f))  # noqa: E731
    if case["kind"] == "traj":
        v = _traj_values(case["T"], gen)
    elif case["kind"] == "kkt":  # 7-point Hessian plus a barrier diagonal, N(0, 1) constraint rows
        v = torch.cat([6.0 + u(p.nh, -8.0, 8.0), -torch.ones(p.edges, **f),
                       torch.randn(4 * case["cons"], generator=gen, **f), torch.full((case["cons"],), -1e-8, **f)])
    elif case["kind"] == "grid2":  # 5-point Laplacian plus a barrier diagonal
        v = torch.cat([4.0 + u(p.n, -8.0, 0.0), -torch.ones(p.ea.numel(), **f)])
    else:  # 7-point operator of log-uniform conductivities
        c = u(p.ea.numel(), -3.0, 3.0)
        d = torch.full((p.n,), 1e-6, **f)
        # the lists of one direction hold each node at most once: the order of
        # these sums is the same on every call
        lo = 0
        for count in _axis_counts(case):
            for e in (p.ea, p.eb):
                d[e[lo:lo + count]] += c[lo:lo + count]
            lo += count
        v = torch.cat([d, -c])
    return v[p.order].contiguous()


def _axis_counts(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    return [nx * ny * (nz - 1), nx * (ny - 1) * nz, (nx - 1) * ny * nz]  # as _grid_edges lists them


def _inputs(case, seed):
    """(values, right-hand sides) on the GPU; a batch's lie one after another."""
    gen = _gen(seed)
    if case["kind"] == "batch":
        hs = _horizons(case)
        v = torch.cat([_traj_values(T, gen)[_traj(T).order] for T in hs])
        n = sum(_traj(T).n for T in hs)
    else:
        p = _pattern(case)
        v, n = _values(case, p, gen), p.n
    b = torch.randn(case["nrhs"], n, dtype=torch.float64, device=DEV, generator=gen)
    return v, b if case["nrhs"] > 1 else b[0].contiguous()


@functools.lru_cache(maxsize=None)
def _traj_analysis(T):
    p = _traj(T)
    return smfg.analyse(p.n, p.ptr, p.idx)


@functools.lru_cache(maxsize=4)
def _analysis(key):
    case = dict(key)
    p = _pattern(case)
    return smfg.analyse(p.n, p.ptr, p.idx)


def _analysis_of(case):
    if case["kind"] == "batch":
        return [_traj_analysis(T) for T in _horizons(case)]
    keep = ("kind", "T", "m", "cons", "nx", "ny", "nz")
    return _analysis(tuple((k, case[k]) for k in keep if k in case))


def _factor_options(case):
    o = {"posdef": case["kind"] in ("grid2", "grid3"), "graph": bool(case.get("graph"))}
    if case["kind"] == "kkt":
        o["aptp_min_rows"] = smfg.APTP_MIN_ROWS if case["aptp"] else 0
    if case.get("mixed"):
        o["precision"] = smfg.PREC_MIXED
        o["mixed_kind"] = smfg.TC_TF32X3 if case["mixed"] == "tf32" else smfg.TC_BF16X3
    return o


# ---------------------------------------------------------------------------


class State:
    pass


def prepare(case, seed):
    s = State()
    s.case, s.nrhs = case, case["nrhs"]
    s.v, s.b = _inputs(case, seed)
    s.opt = _factor_options(case)
    an = _analysis_of(case)
    scale = None
    if case["kind"] == "kkt":  # an interior-point session keeps the scaling of its first values
        p = _pattern(case)
        scale = smfg.matching_scale(p.n, p.ptr, p.idx, s.v.cpu().numpy())[0]
    if case.get("host"):
        s.v, s.b = (t.cpu().pin_memory().numpy() for t in (s.v, s.b))
    if case["kind"] == "batch":
        s.batch = batch.BatchSolver(an, device=0)
        s.solver = s.batch
    elif case.get("session"):
        s.solver = ipm.IpmSession(device=0)
        s.solver.analyse(an, scale=scale, aptp_min_rows=s.opt["aptp_min_rows"])
    else:
        s.solver = smfg.Solver(an, device=0)
        s.opt["scale"] = scale
    if case["do"] == "solve":
        s.solver.factor(s.v, **s.opt)
    return s


def run(s):
    case = s.case
    out = {}
    if case.get("session"):
        s.solver.factor(s.v)
        out["x"], _ = s.solver.solve(s.b)
        out["inertia"] = list(s.solver.inertia())
        return out
    if case["do"] != "solve":
        info = s.solver.factor(s.v, **s.opt)
        out["inertia"] = list(info.inertia)
    if case.get("host"):
        x = s.solver.solve(s.b)
        if case["do"] == "refine":
            x = s.solver.refine(s.b, x, omega_target=OMEGA, method=smfg.REFINE_AUTO, inplace=True)[0]
    else:
        x = s.solver.solve(s.b.clone())
        if case["do"] == "refine":
            sv = s.batch.solver if case["kind"] == "batch" else s.solver
            sv.refine_device(s.b, x, nrhs=s.nrhs, omega_target=OMEGA, method=smfg.REFINE_AUTO)
    out["x"] = x
    return out


def work(case):
    """Values read, L written once and read by both sweeps of the solve, the
    vectors; the delay-free elimination and the sweeps' products."""
    ans = _analysis_of(case)
    by = fl = 0.0
    for a in ans if isinstance(ans, list) else [ans]:
        w = (a.sn_end - a.sn_start).astype(np.float64)
        f = np.diff(a.front_row_ptr).astype(np.float64)
        q = f - w
        entries = float(np.sum(f * f - q * q + w)) / 2
        sq = lambda m: m * (m + 1) * (2 * m + 1) / 6  # noqa: E731
        factor = float(np.sum(sq(f - 1) - sq(q - 1) * (q > 0)))
        nnz = float(a.perm_col_ptr[-1])
        if case["do"] != "solve":
            by += 12 * nnz + 8 * entries
            fl += factor
        by += 16 * entries + 16.0 * a.n * case["nrhs"]
        fl += 4 * entries * case["nrhs"]
        if case["do"] == "refine":  # at least one residual
            by += 24 * nnz + 24.0 * a.n * case["nrhs"]
            fl += 4 * nnz * case["nrhs"]
    return {"bytes": by, "flops": fl}


def tolerance(case):
    """Solutions of the same system by another order of the same 64-bit sums
    differ by rounding times the condition number, which differs by family:
    about four times the largest error seen against exact() over seventy drawn
    cases and the listed ones (the 7-point operator is singular but for its
    1e-6 shift; its largest error was 5e-8, the others' 3e-13)."""
    if case["kind"] == "grid3":
        return {"rel": 2e-7, "max": 4e-7}
    if case["kind"] == "grid2":
        return {"rel": 1e-13, "max": 1e-12}
    return {"rel": 2e-12, "max": 2e-11}


# ---------------------------------------------------------------------------
# The solutions in 64 bits by plain torch: dense factorizations where the
# order allows, conjugate gradients on the larger grids.


def _dense(p, v):
    A = torch.zeros(p.n, p.n, dtype=torch.float64, device=DEV)
    r, c = torch.from_numpy(p.rows).to(DEV), torch.from_numpy(p.cols).to(DEV)
    A[r, c] = v
    A[c, r] = v
    return A


def _dense_solve(p, v, b):
    """LU with equilibration and iterative refinement; b (nrhs, n)."""
    A = _dense(p, v)
    s = 1.0 / A.abs().amax(1).sqrt()
    lu, piv = torch.linalg.lu_factor(A * s[:, None] * s[None, :])
    x = torch.zeros_like(b)
    for _ in range(4):
        r = b - x @ A
        x = x + (torch.linalg.lu_solve(lu, piv, (r * s).T) * s[:, None]).T
    return x


def _grid_solve(p, v, b):
    """Conjugate gradients with a diagonal preconditioner, restarted on the
    true residual; one right-hand side b (n)."""
    r, c = torch.from_numpy(p.rows).to(DEV), torch.from_numpy(p.cols).to(DEV)
    off = r != c
    A = torch.sparse_coo_tensor(torch.stack([torch.cat([r, c[off]]), torch.cat([c, r[off]])]),
                                torch.cat([v, v[off]]), (p.n, p.n)).to_sparse_csr()
    dinv = 1.0 / v[~off]
    x = torch.zeros_like(b)
    for _ in range(4):
        res = b - A @ x
        d = torch.zeros_like(b)
        z = dinv * res
        q, rz, stop = z.clone(), res @ z, 1e-13 * float(res.norm())
        for it in range(20000):
            Aq = A @ q
            a = rz / (q @ Aq)
            d += a * q
            res = res - a * Aq
            z = dinv * res
            new = res @ z
            q = z + (new / rz) * q
            rz = new
            if it % 50 == 49 and float(res.norm()) <= stop:
                break
        x = x + d
    return x


def exact(case, seed):
    v, b = _inputs(case, seed)
    if case["kind"] == "batch":
        x, o, e = torch.empty_like(b), 0, 0
        for T in _horizons(case):
            p = _traj(T)
            cols, ents = slice(o, o + p.n), slice(e, e + p.ptr[-1])
            x[..., cols] = _dense_solve(p, v[ents], b[..., cols].reshape(-1, p.n)).reshape(b[..., cols].shape)
            o, e = cols.stop, int(ents.stop)
    else:
        p = _pattern(case)
        if p.n <= 24000:
            x = _dense_solve(p, v, b.reshape(-1, p.n)).reshape(b.shape)
        elif case["nrhs"] == 1:
            x = _grid_solve(p, v, b)
        else:
            return None
    x = x.cpu().numpy() if case.get("host") else x
    if case["do"] == "solve":
        return {"x": x}
    return {"inertia": None, "x": x}
