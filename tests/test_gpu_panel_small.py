"""Narrow cblks at the edges of k_panel_small: widths around its two rows per
lane and four columns per step, and numbers of off-diagonal bloks around the
tables it keeps (128 bloks, 1024 pairs of bloks: 45 bloks fill them at once,
one blok of 1100 overflows them alone).

Leaves of w columns face scattered single rows of one dense trailing
supernode.  Bar: the backward error of a stable solve, n u = 3e-13.
"""
from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sps

from conftest import FACT_ID, backward_error
from pastix_b200 import gen
from pastix_b200 import pastix as px
from pastix_b200.spm import mtxtype, spmatrix

pytestmark = pytest.mark.gpu


def _leaves(w, bloks, trailing, sym, seed=0):
    """Three leaves of w columns, each joined to `bloks` rows of the trailing block, no two adjacent."""
    rng = np.random.default_rng(seed)
    n = 3 * w + trailing
    M = np.zeros((n, n))
    M[3 * w:, 3 * w:] = rng.uniform(-1, 1, (trailing, trailing))
    for q in range(3):
        c = slice(q * w, (q + 1) * w)
        rows = 3 * w + 2 * np.sort(rng.choice(trailing // 2, bloks, replace=False))
        M[c, c] = rng.uniform(-1, 1, (w, w))
        M[rows, c] = rng.uniform(-1, 1, (bloks, w))
        M[c, rows] = rng.uniform(-1, 1, (w, bloks))
    if sym:
        M = np.tril(M) + np.tril(M, -1).T
    M[np.arange(n), np.arange(n)] = 1.0 + np.abs(M).sum(axis=1)
    rang = np.array([0, w, 2 * w, 3 * w, n], dtype=np.int64)
    return sps.csc_matrix(M), rang, np.array([3, 3, 3, -1], dtype=np.int64)


@pytest.mark.parametrize("fact", ["POTRF", "SYTRF", "GETRF"])
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("w,bloks,trailing", [(1, 3, 60), (5, 45, 100), (4, 46, 100), (3, 129, 300), (1, 1100, 2300),
                                              (31, 20, 90), (32, 33, 90), (33, 40, 90), (60, 5, 70)])
def test_narrow_panels(lib, fact, mixed, w, bloks, trailing):
    A, rang, tree = _leaves(w, bloks, trailing, fact != "GETRF")
    n = A.shape[0]
    assert (w + bloks) * w <= 4096  # the leaves are narrow panels
    ip, dp = px.initParam()
    ip[px.iparm.factorization] = FACT_ID[fact]
    ip[px.iparm.mixed] = int(mixed)
    pd = px.init(ip, dp)
    S = spmatrix(A, mtxtype.General if fact == "GETRF" else mtxtype.Symmetric)
    px.subtask_order(pd, S, np.arange(n), rang, tree)
    px.subtask_symbfact(pd)
    px.subtask_blend(pd)
    info = px.solver_info(pd)
    widths = info["cb_lcol"] - info["cb_fcol"] + 1
    assert (widths[:3] == w).all() and int(info["cb_fblok"][1]) - 1 >= bloks
    px.task_numfact(pd, S)
    b = S.full() @ gen.rhs_uniform(n, 1, 2)[:, 0]
    x = b.copy()
    px.task_solve(pd, S, x)
    assert backward_error(S.full(), x, b) < (n * 2.0 ** -24 if mixed else 3e-13)
    px.finalize(pd)
