"""The front kernels by size class on a B200, bit for bit against the oracle:
single dense fronts at the edges of the classes, SPD and indefinite (zero
diagonal blocks force 2x2 pivots and failing candidates), a front with more
children than the fused kernel describes at a time, chains of fronts that
delay columns, a matrix that is not positive definite, and a blocked size
below the fused kernel's.
"""
import ctypes as C

import numpy as np
import pytest

from opt_solver_b200 import smfg
from opt_solver_b200 import workloads as W
from oracle import oracle as O
from tests.cases import dense_lower

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _built(oracle_lib):
    return oracle_lib


def _spd(n, rng):
    G = rng.standard_normal((n, n))
    return G @ G.T + n * np.eye(n)


def _indefinite(n, rng):
    """Mixed signs, a third of the diagonal zero, some zero entries."""
    A = rng.standard_normal((n, n))
    A = A + A.T
    A[rng.random((n, n)) < 0.2] = 0.0
    A = np.tril(A) + np.tril(A, -1).T
    z = rng.permutation(n)[: n // 3]
    A[z, z] = 0.0
    return A


def _compare(a, sv, info, v, posdef, scale=None, **oracle_kw):
    ox = O.restated_factorize(a, O.permuted_values(a, v, scale), posdef, **oracle_kw)
    gx = sv.export()
    assert info.delayed_pivots == ox.delayed and info.two_by_two_pivots == ox.two_by_two
    assert info.flops == ox.flops
    if not posdef:
        assert info.inertia == ox.inertia
    for s in range(a.nsn):
        assert gx.f[s] == ox.f[s] and gx.p[s] == ox.p[s], s
        assert np.array_equal(gx.front_rows(s), ox.front_rows(s)), s
        assert np.array_equal(gx.block(s), ox.block(s)), s
    if not posdef:
        nt = int(np.sum(gx.p))
        assert np.array_equal(gx.tags[:nt], ox.tags[:nt])


def _run(n, cp, ri, v, posdef, nemin=8, ordering=smfg.ORDER_ND):
    a = smfg.analyse(n, cp, ri, ordering=ordering, nemin=nemin)
    sv = smfg.Solver(a, device=0)
    info = sv.factor(v, posdef=posdef)
    _compare(a, sv, info, v, posdef)
    sv.close()
    return a, info


@pytest.mark.parametrize("n", [1, 2, 3, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129])
@pytest.mark.parametrize("posdef", [True, False])
def test_dense_front(n, posdef):
    rng = np.random.default_rng(1000 + n)
    A = _spd(n, rng) if posdef else _indefinite(n, rng)
    a, _ = _run(*dense_lower(A), posdef, ordering=smfg.ORDER_NATURAL)
    assert int(np.diff(a.front_row_ptr).max()) == n


@pytest.mark.parametrize("posdef", [True, False])
def test_many_children(posdef):
    """40 leaves of one column under one root: three batches of children."""
    rng = np.random.default_rng(5)
    k, m = 40, 12
    n = k + m
    A = np.zeros((n, n))
    A[k:, k:] = _spd(m, rng) if posdef else _indefinite(m, rng)
    A[k:, :k] = rng.standard_normal((m, k))
    A[:k, k:] = A[k:, :k].T
    A[np.arange(k), np.arange(k)] = 4.0 * n if posdef else rng.standard_normal(k)
    A[np.arange(k, n), np.arange(k, n)] += 4.0 * n if posdef else 0.0
    rows, cols = np.nonzero(np.tril(A))
    keep = (rows >= k) | (rows == cols)
    rows, cols = rows[keep], cols[keep]
    order = np.lexsort((rows, cols))
    cp = np.zeros(n + 1, np.int32)
    np.add.at(cp, cols + 1, 1)
    a, _ = _run(n, np.cumsum(cp).astype(np.int32), rows[order].astype(np.int32), A[rows, cols][order], posdef,
                nemin=1, ordering=smfg.ORDER_NATURAL)
    assert int(np.diff(a.child_ptr).max()) > 32


@pytest.mark.parametrize("T", [3, 30, 90])
def test_delaying_chain(T):
    n, cp, ri, v = W.trajectory_kkt(T, np.random.default_rng(T))
    _, info = _run(n, cp, ri, v, False)
    assert info.delayed_pivots > 0 and info.two_by_two_pivots > 0


def test_grid_levels():
    _run(*W.laplacian_2d(61, 47), True)


def test_not_positive_definite():
    A = _spd(50, np.random.default_rng(2))
    A[37, 37] = -1.0
    n, cp, ri, v = dense_lower(A)
    a = smfg.analyse(n, cp, ri)
    sv = smfg.Solver(a, device=0)
    info = sv.factor(v, posdef=True)
    assert info.factor_status == smfg.SMFG_FACTOR_NOT_POSDEF
    sv.close()


def _factor(sv, v, posdef, rcs=(smfg.SMFG_OK, smfg.SMFG_ERR_SINGULAR), **fields):
    """Factorization through the C entry with fields of the control set."""
    c = smfg.default_control(posdef)
    for k, x in fields.items():
        setattr(c, k, x)
    info = smfg.Info()
    val = np.ascontiguousarray(v)
    rc = smfg.lib().smfg_factor(sv._h, val.ctypes.data, C.byref(c), C.byref(info))
    assert rc in rcs
    sv.posdef, sv.info = posdef, info
    return info


@pytest.mark.parametrize("blocked", [1, 2, 33, 130])
@pytest.mark.parametrize("kind", ["chain", "grid"])
def test_blocked_min_front_tree(blocked, kind):
    """The same on trees: from the first row on (no front is assembled by its
    own block), with delayed columns and contribution blocks on both sides of
    the edge."""
    posdef = kind == "grid"
    n, cp, ri, v = W.laplacian_2d(121, 97) if posdef else W.trajectory_kkt(200, np.random.default_rng(30))
    a = smfg.analyse(n, cp, ri)
    sv = smfg.Solver(a, device=0)
    info = _factor(sv, v, posdef, blocked_min_front=blocked)
    assert posdef or info.delayed_pivots > 0
    assert info.max_front > 96
    _compare(a, sv, info, v, posdef, blocked_min_front=blocked)
    sv.close()


@pytest.mark.parametrize("blocked", [20, 40, 96, 200])
@pytest.mark.parametrize("posdef", [True, False])
def test_blocked_min_front(blocked, posdef):
    """A blocked size below or above the default moves the classes' edges."""
    rng = np.random.default_rng(8)
    for n in (19, 20, 39, 40, 70, 96, 100):
        A = _spd(n, rng) if posdef else _indefinite(n, rng)
        n, cp, ri, v = dense_lower(A)
        a = smfg.analyse(n, cp, ri, ordering=smfg.ORDER_NATURAL)
        sv = smfg.Solver(a, device=0)
        c = smfg.default_control(posdef)
        c.blocked_min_front = blocked
        info = smfg.Info()
        val = np.ascontiguousarray(v)
        rc = smfg.lib().smfg_factor(sv._h, val.ctypes.data, C.byref(c), C.byref(info))
        assert rc in (smfg.SMFG_OK, smfg.SMFG_ERR_SINGULAR)
        sv.posdef, sv.info = posdef, info
        _compare(a, sv, info, v, posdef, blocked_min_front=blocked)
        sv.close()


@pytest.mark.parametrize("nrhs", [1, 2, 3, 5, 8, 9])
@pytest.mark.parametrize("posdef", [True, False])
def test_solve_by_class(nrhs, posdef):
    """Solves of single dense fronts at the edges of the solve kernels' sizes
    against dense solutions, and the sweeps one by one against the full solve.
    Both are backward stable: |x - y| <= 2 (3 n eps g) cond(A) |x|, with g = 1
    for Cholesky and at most 1 / u growth per pivot bound u = 0.01."""
    rng = np.random.default_rng(40 + nrhs)
    eps = np.finfo(float).eps
    for n in (1, 2, 31, 32, 33, 64, 65, 96, 97, 160, 383, 384, 700):
        A = _spd(n, rng) if posdef else _indefinite(n, rng) + np.diag(np.full(n, 0.5))
        n, cp, ri, v = dense_lower(A)
        sv = smfg.Solver(smfg.analyse(n, cp, ri, ordering=smfg.ORDER_NATURAL), device=0)
        sv.factor(v, posdef=posdef, aptp_min_rows=0)
        b = rng.standard_normal((nrhs, n)) if nrhs > 1 else rng.standard_normal(n)
        want = np.linalg.solve(A, b.T).T
        x = sv.solve(b)
        tol = 6 * n * eps * np.linalg.cond(A) * (1.0 if posdef else 100.0)
        assert np.max(np.abs(x - want)) <= tol * np.max(np.abs(want)), n
        y = sv.solve(sv.solve(sv.solve(b, smfg.SOLVE_FORWARD), smfg.SOLVE_DIAGONAL), smfg.SOLVE_BACKWARD)
        assert np.max(np.abs(y - want)) <= tol * np.max(np.abs(want)), n
        sv.close()


@pytest.mark.parametrize("nrhs", [1, 4, 7])
@pytest.mark.parametrize("kind", ["grid", "chain"])
def test_solve_trees(kind, nrhs):
    """Trees with leaves, tiny and medium fronts, with and without delays: the
    backward error the refinement gate reads (componentwise, 1e-12 after one
    step of refinement at most), and the single columns' solutions."""
    n, cp, ri, v = W.laplacian_2d(83, 71) if kind == "grid" else W.trajectory_kkt(60, np.random.default_rng(1))
    sv = smfg.Solver(smfg.analyse(n, cp, ri), device=0)
    sv.factor(v, posdef=kind == "grid")
    b = np.random.default_rng(2).standard_normal((nrhs, n))
    x = sv.solve(b if nrhs > 1 else b[0]).reshape(nrhs, n)
    for r in range(nrhs):
        one = sv.solve(b[r])
        assert np.max(np.abs(one - x[r])) <= 1e-10 * np.max(np.abs(one))
        _, _, om, steps = sv.refine(b[r], one, omega_target=1e-12)
        assert om <= 1e-12 and steps <= 1
    sv.close()


@pytest.mark.parametrize("n,ne", [(330, 130), (520, 260), (700, 77)])
@pytest.mark.parametrize("kind", ["wide", "zeros", "subnormal"])
def test_schur_matrix_instructions(n, ne, kind):
    """The contribution block of a large front against chains of fused
    multiply-adds in pivot order (the oracle's): odd sizes, chunks with and
    without zero multipliers, a wide range of magnitudes, and entries down to
    the subnormal numbers."""
    rng = np.random.default_rng(n)
    A = _spd(n, rng)
    s = np.full(n, 1e-155) if kind == "subnormal" else 10.0 ** rng.uniform(-6, 6, n)
    if kind == "zeros":  # rows without entries in some of the pivots' columns
        A[ne:, : ne // 2] *= rng.random((n - ne, 1)) < 0.6
        A[: ne // 2, ne:] = A[ne:, : ne // 2].T
        A[np.arange(n), np.arange(n)] += n
    A = A * s[:, None] * s[None, :]
    n, cp, ri, v = dense_lower(A)
    # two supernodes: the first ne columns, whose update the second takes
    a = smfg.analyse(n, cp, ri, ordering=smfg.ORDER_NATURAL)
    arrays = {k: getattr(a, k).copy() for k in smfg._ANALYSIS_FIELDS}
    arrays["sn_start"], arrays["sn_end"] = np.int32([0, ne]), np.int32([ne, n])
    arrays["sn_parent"], arrays["postorder"] = np.int32([1, -1]), np.int32([0, 1])
    arrays["child_ptr"], arrays["child_idx"] = np.int32([0, 0, 1]), np.int32([0])
    arrays["front_row_ptr"] = np.int32([0, n, 2 * n - ne])
    arrays["front_row_idx"] = np.concatenate([np.arange(n), np.arange(ne, n)]).astype(np.int32)
    b = smfg.Analysis(n, arrays)
    for posdef in (True,) if kind == "subnormal" else (True, False):
        sv = smfg.Solver(b, device=0)
        info = sv.factor(v, posdef=posdef, aptp_min_rows=0)
        _compare(b, sv, info, v, posdef, aptp_min_rows=0)
        sv.close()


@pytest.mark.parametrize("n,bad", [(300, 36), (300, 37), (300, 143), (96, 51), (97, 50)])
def test_not_positive_definite_large(n, bad):
    """A pivot that fails at an even or odd place of a pair, in the first or the
    second panel of a step: the columns before it are those of the matrix that
    differs from it in that diagonal entry alone, the run on the static layout
    is given up and redone, and the next factorization of the plan is
    unaffected."""
    rng = np.random.default_rng(n + bad)
    A = _spd(n, rng)
    good = dense_lower(A)
    A[bad, bad] = -5.0
    _, cp, ri, v = dense_lower(A)
    a = smfg.analyse(n, cp, ri, ordering=smfg.ORDER_NATURAL)
    sv = smfg.Solver(a, device=0)
    for _ in range(2):
        info = sv.factor(v, posdef=True)
        assert info.factor_status == smfg.SMFG_FACTOR_NOT_POSDEF
        stopped = sv.export().block(0)[:, :bad]
        gi = sv.factor(good[3], posdef=True)
        _compare(a, sv, gi, good[3], True)
        assert np.array_equal(stopped, sv.export().block(0)[:, :bad])
    sv.close()


@pytest.mark.parametrize("m", [6, 12, 20])
def test_not_positive_definite_tree(m):
    """Failed pivots all over a tree: the columns they delay grow the fronts
    above past their symbolic size class, and the factorization still reports
    NOT_POSDEF, twice the same; the next one of good values is the oracle's."""
    n, cp, ri, good = W.varcoef_3d(m, seed=m)
    v = good.copy()
    v[W.diagonal_slots(n, cp, ri)[np.random.default_rng(m).choice(n, 3)]] *= -1
    a = smfg.analyse(n, cp, ri)
    sv = smfg.Solver(a, device=0)
    runs = []
    for _ in range(2):
        info = sv.factor(v, posdef=True)
        assert info.factor_status == smfg.SMFG_FACTOR_NOT_POSDEF
        assert sum(info.inertia) + info.delayed_pivots >= n
        runs.append((info.inertia, info.delayed_pivots, info.flops, sv.front_stats().tolist()))
    assert runs[0] == runs[1]
    assert runs[0][1] > 0
    gi = sv.factor(good, posdef=True)
    _compare(a, sv, gi, good, True)
    sv.close()


def test_panel_width_changes():
    """One SPD plan factored with panels of several widths, profiled or not: the
    layout that is kept between factorizations has room for the panel of each
    (width 16 profiled and width 32 give the large fronts as many rows of W).
    Every factor is that of a plan of its own, bit for bit. The
    fronts include some of 129..191 rows, which one block factors in global
    memory, several on a level."""
    n, cp, ri, v = W.varcoef_3d(14, seed=3)
    a = smfg.analyse(n, cp, ri)
    rows = np.diff(a.front_row_ptr)
    assert np.sum((rows > 128) & (rows < 192)) >= 4 and rows.max() >= 192
    sv = smfg.Solver(a, device=0)
    for nb, profile in ((16, 0), (48, 0), (16, 0), (16, 1), (32, 0), (16, 1), (5, 0), (32, 0)):
        _factor(sv, v, True, nb=nb, profile=profile)
        own = smfg.Solver(a, device=0)
        _factor(own, v, True, nb=nb, profile=profile)
        gx, wx = sv.export(), own.export()
        assert np.array_equal(gx.blocks, wx.blocks) and np.array_equal(gx.rows, wx.rows), (nb, profile)
        own.close()
    sv.close()


@pytest.mark.parametrize("nb", [2, 48, 49, 54, 55, 57])
@pytest.mark.parametrize("posdef", [True, False])
def test_panel_widths(nb, posdef):
    """Panels up to the widest that fits beside a front of 128 rows in shared
    memory (57; from 49 on the front is not padded), bit for bit."""
    rng = np.random.default_rng(nb)
    for n in (97, 127, 128, 129):
        A = _spd(n, rng) if posdef else _indefinite(n, rng)
        n, cp, ri, v = dense_lower(A)
        a = smfg.analyse(n, cp, ri, ordering=smfg.ORDER_NATURAL)
        sv = smfg.Solver(a, device=0)
        info = _factor(sv, v, posdef, nb=nb)
        _compare(a, sv, info, v, posdef, nb=nb)
        sv.close()


def _spd_report(a, v):
    """What a factorization without pivoting finds when pivots may fail: the
    columns from a front's first failed pivot on are delayed to its parent.
    Per supernode (rows, pivots, delayed columns, flops); plain numpy."""
    pv = O.permuted_values(a, v)
    out, cb = np.zeros((a.nsn, 4)), {}
    for s in a.postorder:
        kids = a.child_idx[a.child_ptr[s]:a.child_ptr[s + 1]]
        rows = [r for c in kids for r in cb[c][1]]
        ne = len(rows) + a.sn_end[s] - a.sn_start[s]
        rows += list(a.front_row_idx[a.front_row_ptr[s]:a.front_row_ptr[s + 1]])
        pos = {r: i for i, r in enumerate(rows)}
        f = len(rows)
        F = np.zeros((f, f))
        for j in range(a.sn_start[s], a.sn_end[s]):
            for k in range(a.perm_col_ptr[j], a.perm_col_ptr[j + 1]):
                F[pos[a.perm_row_idx[k]], pos[j]] += pv[k]
        for c in kids:
            m, _, r = cb.pop(c)
            ix = np.array([pos[x] for x in r], dtype=np.int64)
            F[np.ix_(ix, ix)] += m
        p, fl = 0, 0.0
        while p < ne and F[p, p] > 0.0:
            F[p + 1:, p + 1:] -= np.outer(F[p + 1:, p], F[p + 1:, p] / F[p, p])
            p += 1
            fl += (f - p) + (f - p) * (f - p + 1.0)
        root = a.sn_parent[s] < 0
        out[s] = f, p, 0 if root else ne - p, fl
        cb[s] = (np.tril(F[p:, p:]), [] if root else rows[p:ne], [] if root else rows[p:])
    return out


@pytest.mark.parametrize("m,bad", [(6, 1), (12, 1), (12, 3), (16, 2), (20, 1), (20, 4)])
def test_not_positive_definite_report(m, bad):
    """Counts, sizes and delays of a factorization that fails, whether it goes on
    from the level that failed (from the second call on, and after a replay) or
    is redone whole (the first, whose arena has no room; a profiled one)."""
    import torch
    n, cp, ri, good = W.varcoef_3d(m, seed=m)
    v = good.copy()
    v[W.diagonal_slots(n, cp, ri)[np.random.default_rng(m).choice(n, bad)]] *= -1
    a = smfg.analyse(n, cp, ri)
    want = _spd_report(a, v)
    sv = smfg.Solver(a, device=0)
    own = smfg.Solver(a, device=0)
    own.factor(good, posdef=True)
    blocks = own.export().blocks
    d_v = torch.from_numpy(good.copy()).cuda()
    rcs = (smfg.SMFG_ERR_SINGULAR,)
    for how in ("plain", "plain", "profile", "plain", "graph", "plain"):
        if how == "graph":
            for values in (good, v):  # captured, then replayed
                d_v.copy_(torch.from_numpy(values))
                info = sv.factor(d_v, posdef=True, graph=True)
        else:
            info = _factor(sv, v, True, rcs=rcs, profile=int(how == "profile"))
        assert info.factor_status == smfg.SMFG_FACTOR_NOT_POSDEF
        gx, st = sv.export(), sv.front_stats()
        assert np.array_equal(gx.f, want[:, 0]), how
        assert np.array_equal(st[:, 0], want[:, 1]) and np.array_equal(st[:, 4], want[:, 2]), how
        assert info.flops == want[:, 3].sum() and info.delayed_pivots == want[:, 2].sum()
        assert info.max_front == want[:, 0].max()
        assert info.inertia == (want[:, 1].sum(), 0, n - want[:, 1].sum())
        # a front with delayed columns takes no pivot: the first is the failed one
        assert not np.any(want[want[:, 0] > np.diff(a.front_row_ptr), 1])
        sv.factor(good, posdef=True)
        assert np.array_equal(sv.export().blocks, blocks)
    sv.close()
    own.close()


def _leaves_under_root(k, m, posdef, rng):
    """k leaves of one column, whose contribution blocks cover a dense root of m
    columns (natural order)."""
    n = k + m
    A = np.zeros((n, n))
    A[k:, k:] = _spd(m, rng) if posdef else _indefinite(m, rng)
    A[k:, :k] = rng.standard_normal((m, k))
    A[np.arange(k), np.arange(k)] = 4.0 * n if posdef else 1.0 + rng.random(k)
    if posdef:
        A[np.arange(k, n), np.arange(k, n)] += 4.0 * n
    rows, cols = np.nonzero(np.tril(A))
    order = np.lexsort((rows, cols))
    cp = np.concatenate([[0], np.cumsum(np.bincount(cols, minlength=n))])
    return n, cp.astype(np.int32), rows[order].astype(np.int32), A[rows, cols][order]


@pytest.mark.parametrize("k,m", [(16, 110), (17, 110), (40, 100), (40, 250), (16, 768), (16, 769), (13, 946)])
@pytest.mark.parametrize("posdef", [True, False])
def test_assembly_maps(k, m, posdef):
    """Assembly of a front past the fused sizes on both sides of the room for its
    children's inverse row maps (16 children, children x rows 12,288): gathered,
    or a pass per child."""
    # (the last leaf is merged into the root)
    a, _ = _run(*_leaves_under_root(k + 1, m - 1, posdef, np.random.default_rng(k + m)), posdef, nemin=1,
                ordering=smfg.ORDER_NATURAL)
    assert int(np.diff(a.child_ptr).max()) == k and int(np.diff(a.front_row_ptr).max()) == m


@pytest.mark.parametrize("n", [1, 20, 32, 33, 64])
@pytest.mark.parametrize("nrhs", [1, 5])
def test_small_solves_divide(n, nrhs):
    """SPD fronts of up to 64 rows divide by the diagonal of L (a rounded
    reciprocal and its correction): a diagonal matrix in one dense front is
    solved as plain divisions round it, infinities as divisions leave them."""
    rng = np.random.default_rng(n)
    d = 10.0 ** rng.uniform(-8, 8, n)
    _, cp, ri, v = dense_lower(np.diag(d))
    sv = smfg.Solver(smfg.analyse(n, cp, ri, ordering=smfg.ORDER_NATURAL), device=0)
    sv.factor(v, posdef=True)
    b = rng.standard_normal((nrhs, n)) * 10.0 ** rng.uniform(-100, 100, (nrhs, n))
    b[0, 0] = np.inf
    l = np.sqrt(d)
    x = sv.solve(b if nrhs > 1 else b[0]).reshape(nrhs, n)
    assert np.array_equal(x, (b / l) / l)
    sv.close()
