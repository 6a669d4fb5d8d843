"""CUDA-graph replay of the factorization (smfg_control_t.graph): the first
call captures, later calls with the same configuration replay; a replay
gives the normal path's factor bit for bit, also on new values of the same
pattern (the interior-point refactor), and falls back to the normal path
when the configuration changes."""
import numpy as np
import pytest

from opt_solver_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["spd", "kkt", "kkt_mixed"])
def test_graph_replay_bitwise(kind):
    import torch
    from opt_solver_b200 import smfg
    if kind == "spd":
        n, cp, ri, v = W.varcoef_3d(20, seed=2)
        posdef = True
    else:
        n, cp, ri, v = W.kkt_ipm(12, 800, seed=4)
        posdef = False
    prec = smfg.PREC_MIXED if kind == "kkt_mixed" else smfg.PREC_FP64
    a = smfg.analyse(n, cp, ri)
    sv = smfg.Solver(a, device=0)
    d_v = torch.from_numpy(np.ascontiguousarray(v)).cuda()
    ref = sv.factor(d_v, posdef=posdef, precision=prec)
    e_ref = sv.export()
    g1 = sv.factor(d_v, posdef=posdef, precision=prec, graph=True)   # normal + capture
    g2 = sv.factor(d_v, posdef=posdef, precision=prec, graph=True)   # replay
    e2 = sv.export()
    assert g2.inertia == ref.inertia and g2.delayed_pivots == ref.delayed_pivots
    assert np.array_equal(e2.blocks, e_ref.blocks) and np.array_equal(e2.rows, e_ref.rows)
    # new values of the same pattern (a scaled diagonal), replayed in place
    # (SPD: a larger diagonal keeps it positive definite; KKT: the primal
    # block's diagonal, Sigma, moves as in an interior-point iteration)
    rng = np.random.default_rng(1)
    v2 = v.copy()
    diag = np.asarray(ri) == np.repeat(np.arange(n), np.diff(cp))
    sel = diag & (v > 0)
    v2[sel] *= rng.uniform(1.0, 2.0, int(sel.sum()))
    d_v.copy_(torch.from_numpy(v2))
    g3 = sv.factor(d_v, posdef=posdef, precision=prec, graph=True)   # replay
    e3 = sv.export()
    r3 = sv.factor(d_v, posdef=posdef, precision=prec)               # normal path
    er = sv.export()
    assert g3.inertia == r3.inertia and g3.delayed_pivots == r3.delayed_pivots
    assert np.array_equal(e3.blocks, er.blocks)
    b = W.rhs(n, 1, seed=3)
    x = sv.solve(b)
    x, _, om, _ = sv.refine(b, x, max_steps=20, omega_target=1e-13, method=smfg.REFINE_AUTO)
    assert om < 1e-12
    sv.close()


def _two_supernodes(ne, n, rng):
    """A dense SPD matrix whose first ne columns are one supernode and the rest
    its parent: a pivot that fails in the first delays columns into the second."""
    from opt_solver_b200 import smfg
    from tests.cases import dense_lower
    G = rng.standard_normal((n, n))
    n, cp, ri, v = dense_lower(G @ G.T + n * np.eye(n))
    a = smfg.analyse(n, cp, ri, ordering=smfg.ORDER_NATURAL)
    arrays = {k: getattr(a, k).copy() for k in smfg._ANALYSIS_FIELDS}
    arrays["sn_start"], arrays["sn_end"] = np.int32([0, ne]), np.int32([ne, n])
    arrays["sn_parent"], arrays["postorder"] = np.int32([1, -1]), np.int32([0, 1])
    arrays["child_ptr"], arrays["child_idx"] = np.int32([0, 0, 1]), np.int32([0])
    arrays["front_row_ptr"] = np.int32([0, n, 2 * n - ne])
    arrays["front_row_idx"] = np.concatenate([np.arange(n), np.arange(ne, n)]).astype(np.int32)
    return n, cp, v, smfg.Analysis(n, arrays)


@pytest.mark.parametrize("ne,n", [(10, 38), (40, 130), (70, 230)])
def test_graph_with_failed_pivots(ne, n):
    """Matrices that are not positive definite, with a graph, between good ones
    with and without it. The failed columns are delayed into a parent that
    leaves its size class (28 rows to 34 and more); every good factorization
    is that of a plan of its own, bit for bit, and the graph stays the one of
    good factorizations."""
    import torch
    from opt_solver_b200 import smfg
    n, cp, v, a = _two_supernodes(ne, n, np.random.default_rng(n))
    bad = v.copy()
    bad[cp[4]] = -1.0
    sv, own = smfg.Solver(a, device=0), smfg.Solver(a, device=0)
    own.factor(v, posdef=True)
    want = own.export().blocks
    d_v = torch.from_numpy(v.copy()).cuda()
    reports, launches = [], []
    for values, graph in ((bad, True), (v, False), (bad, True), (v, False), (v, True), (bad, True), (v, True),
                          (bad, False), (v, True), (bad, True), (v, False)):
        d_v.copy_(torch.from_numpy(values))
        info = sv.factor(d_v, posdef=True, graph=graph)
        if values is bad:
            assert info.factor_status == smfg.SMFG_FACTOR_NOT_POSDEF
            assert info.delayed_pivots == ne - 4
            reports.append((info.inertia, info.delayed_pivots, info.flops, info.max_front))
        else:
            assert info.factor_status == smfg.SMFG_FACTOR_SUCCESS
            assert np.array_equal(sv.export().blocks, want)
            launches.append(info.kernel_launches)
    assert all(r == reports[0] for r in reports)
    assert len(set(launches)) == 1  # no good factorization takes the level-by-level kernels
    sv.close()
    own.close()


@pytest.mark.parametrize("m", [12, 20])
def test_kinds_alternate_on_one_plan(m):
    """SPD and indefinite factorizations of one plan in turn, plain and by graph:
    each has its own large fronts, and every factor and solution is that of a
    plan that only ever took its kind, bit for bit."""
    import torch
    from opt_solver_b200 import smfg
    n, cp, ri, v = W.varcoef_3d(m, seed=m)
    a = smfg.analyse(n, cp, ri)
    b = W.rhs(n, 2, seed=3)
    d_v = torch.from_numpy(v.copy()).cuda()
    want = {}
    for posdef in (True, False):
        own = smfg.Solver(a, device=0)
        own.factor(d_v, posdef=posdef)
        want[posdef] = own.export().blocks, own.solve(b)
        own.close()
    sv = smfg.Solver(a, device=0)
    for posdef, graph in ((True, True), (False, False), (True, True), (False, False), (True, False), (False, True),
                          (True, False), (False, True), (True, True), (True, True), (False, False)):
        sv.factor(d_v, posdef=posdef, graph=graph)
        assert np.array_equal(sv.export().blocks, want[posdef][0])
        assert np.array_equal(sv.solve(b), want[posdef][1])
    sv.close()
