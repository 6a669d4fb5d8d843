"""A factorization that is given up in the middle of a tree level: every kernel
takes that decision alike in all threads of a block (a flag may be set while
the block reads it), and what follows is unaffected.
"""
import os
import re

import numpy as np
import pytest

from opt_solver_b200 import build, smfg
from tests.cases import dense_lower


def _kernels():
    """(name, body) of every __global__ function, comments removed."""
    for src in sorted(os.listdir(build.CSRC)):
        with open(os.path.join(build.CSRC, src)) as fh:
            text = re.sub(r"//[^\n]*", "", fh.read())
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\(([^{;]*)\)\s*\{", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            yield m.group(1), text[m.end():i]


def test_abort_decided_per_block():
    """No kernel of more than one working thread reads the abort flags in more
    than one thread of a block, and none that asks block_aborted returns before
    it does."""
    seen = 0
    for name, body in _kernels():
        assert "kFAbort" not in body, name
        if "block_aborted" in body:
            seen += 1
            assert "return" not in body[:body.index("block_aborted")], name
        if "abort_flagged" in body:
            seen += 1
            assert re.search(r"threadIdx\.x == 0 && abort_flagged|^\s*if \(threadIdx\.x != 0", body), name
    assert seen >= 10


def _forest(blocks):
    """Lower CSC of a block-diagonal matrix of dense blocks."""
    parts = [dense_lower(A) for A in blocks]
    off = np.cumsum([0] + [p[0] for p in parts])
    ptr = np.cumsum([0] + [len(p[3]) for p in parts])
    cp = np.concatenate([p[1][:-1] + q for p, q in zip(parts, ptr)] + [ptr[-1:]])
    ri = np.concatenate([p[2] + o for p, o in zip(parts, off)])
    return int(off[-1]), cp.astype(np.int32), ri.astype(np.int32), np.concatenate([p[3] for p in parts])


@pytest.mark.gpu
def test_failed_pivots_beside_other_fronts(oracle_lib):
    """Fronts of every size class on one level, a failing pivot in some of each:
    the classes run side by side, so a flag is set while other fronts are
    assembled, factored and stored. The report is the same every time, and the
    next factorization of good values is the oracle's."""
    from opt_solver_b200 import workloads as W
    O = oracle_lib
    rng = np.random.default_rng(11)
    sizes = np.tile([9, 30, 50, 64, 80, 95, 96, 110, 128, 150, 190, 200, 300, 420], 12)
    blocks = []
    for n in sizes:
        G = rng.standard_normal((n, n))
        blocks.append(G @ G.T + n * np.eye(n))
    n, cp, ri, good = _forest(blocks)
    starts = np.cumsum([0, *sizes[:-1]])
    diag = W.diagonal_slots(n, cp, ri)
    a = smfg.analyse(n, cp, ri, ordering=smfg.ORDER_NATURAL)
    ox = O.restated_factorize(a, O.permuted_values(a, good), True)
    sv = smfg.Solver(a, device=0)
    for trial in range(6):
        v = good.copy()
        hit = rng.random(len(sizes)) < (0.05 if trial % 2 else 0.5)
        hit[0] = True
        for s, m, h in zip(starts, sizes, hit):
            if h:
                v[diag[s + rng.integers(m)]] = -1.0
        runs = []
        for _ in range(4):
            info = sv.factor(v, posdef=True)
            assert info.factor_status == smfg.SMFG_FACTOR_NOT_POSDEF
            runs.append((info.inertia, info.delayed_pivots, info.flops, sv.front_stats().tolist()))
        assert all(r == runs[0] for r in runs)
        sv.factor(good, posdef=True)
        gx = sv.export()
        assert all(np.array_equal(gx.block(f), ox.block(f)) for f in range(a.nsn))
    sv.close()
