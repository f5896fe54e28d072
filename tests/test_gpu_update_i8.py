"""FP64 updates by integer slices on the tensor cores, at the edges of their
tiles: source widths around the 32-column K blocks, bloks and panels that do
not fill the 128 x 128 windows, every factorization kind, matrices whose rows
differ in scale by many orders of magnitude, and a non-finite entry.

Factors against the oracle's: both sum at most n products per entry, so
n u = 4e-13 bounds their difference relative to the factor (observed 1e-15).
"""
from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sps

from conftest import FACT_ID, analyse, backward_error
from pastix_b200 import gen
from pastix_b200 import pastix as px
from pastix_b200.spm import mtxtype, spmatrix
from test_gpu_parity import _mask_compare

pytestmark = pytest.mark.gpu


def _system(fact):
    if fact == "GETRF":
        return gen.convdiff27(15, 14, 13), (15, 14, 13)
    return gen.laplacian7(17, 18, 19), (17, 18, 19)


@pytest.mark.parametrize("fact", ["POTRF", "SYTRF", "GETRF"])
@pytest.mark.parametrize("bs", [(32, 33), (40, 64), (64, 65), (96, 129), (160, 320)])
def test_factors_at_tile_edges(lib, oracle_mod, fact, bs):
    _factors_against_oracle(oracle_mod, fact, bs, True)


@pytest.mark.parametrize("fact", ["POTRF", "SYTRF", "GETRF"])
@pytest.mark.parametrize("bs", [(32, 33), (40, 64), (64, 65), (160, 320)])
def test_fp64_tiles_of_the_same_tasks(lib, oracle_mod, fact, bs):
    """The DMMA tiles that take these tasks where the integer slices cannot be used."""
    _factors_against_oracle(oracle_mod, fact, bs, False)


def _factors_against_oracle(oracle_mod, fact, bs, integer):
    A, grid = _system(fact)
    pd, S, info = analyse(A, grid, fact, min_bs=bs[0], max_bs=bs[1])
    px.integer_updates(pd, integer)
    px.task_numfact(pd, S)
    assert px.get_update_path(pd) == (integer, 0)
    Lg, Ug = px.get_coeftab(pd, with_u=(fact == "GETRF"))
    sym = oracle_mod.Symbol(info)
    Ap = oracle_mod.permuted_full(S.full(), info["permtab"])
    L2, U2, npiv = oracle_mod.factor(sym, Ap, fact, oracle_mod.criterion(Ap))
    assert int(pd.iparm[px.iparm.static_pivoting]) == npiv
    keep = _mask_compare(fact, info)
    Lo = oracle_mod.to_panels(sym, L2)
    assert np.linalg.norm((Lg - Lo)[keep]) / np.linalg.norm(Lo[keep]) < 4e-13
    if fact == "GETRF":
        Uo = oracle_mod.to_panels(sym, U2)
        assert np.linalg.norm(Ug - Uo) / np.linalg.norm(Uo) < 4e-13
    px.finalize(pd)


@pytest.mark.parametrize("fact", ["POTRF", "SYTRF", "GETRF"])
@pytest.mark.parametrize("decades", [8, 100, 250])
def test_scaled_rows(lib, fact, decades):
    """D A D with d spread over many decades: the rounding is relative to each row."""
    A, grid = _system(fact)
    n = A.shape[0]
    d = 10.0 ** np.random.default_rng(1).uniform(-decades / 4, decades / 4, n)
    M = (sps.diags(d) @ A @ sps.diags(d)).tocsc()
    pd, S, info = analyse(M, grid, fact)
    pd.dparm[px.dparm.epsilon_magn_ctrl] = -1e-300  # no pivot is small here
    px.task_numfact(pd, S)
    xt = gen.rhs_uniform(n, 1, 3)[:, 0]
    b = S.full() @ (xt / d)  # solution xt / d
    x = b.copy()
    px.task_solve(pd, S, x)
    # in the unscaled unknowns the backward error is that of a stable solve of A
    assert backward_error(A, d * x, b / d) < 4e-13
    px.finalize(pd)


def _lu_error(M, grid, A, xt, l, r, integer=True, **kw):
    """Relative error in the unscaled unknowns of M = 2^l A 2^r, and the sources handed back to FP64 arithmetic."""
    pd, S, info = analyse(M, grid, "GETRF", **kw)
    pd.dparm[px.dparm.epsilon_magn_ctrl] = -1e-300
    px.integer_updates(pd, integer)
    px.task_numfact(pd, S)
    assert int(pd.iparm[px.iparm.static_pivoting]) == 0
    b = np.ldexp(A @ xt, l)
    px.task_solve(pd, S, b)
    used, flagged = px.get_update_path(pd)
    assert used == integer
    nc, st = info["cb_lcol"] - info["cb_fcol"] + 1, info["cb_stride"]
    sources = int(((nc >= 32) & (nc <= 512) & (nc * st > 4096) & (st > nc)).sum())
    px.finalize(pd)
    return np.linalg.norm(np.ldexp(b, r) - xt) / np.linalg.norm(xt), flagged / sources


@pytest.mark.parametrize("decades", [8, 14, 40, 200])
@pytest.mark.parametrize("kind", ["rows", "columns", "rows and columns", "both alike", "rows of one half"])
def test_lu_of_scaled_rows_and_columns(lib, decades, kind):
    """D1 A D2 with powers of two drawn per row and column: FP64 elimination without pivoting does the same
    arithmetic for every such scaling, so the error in the unscaled unknowns is that of A itself (twice that is
    allowed for the order of the scattered sums)."""
    A, grid = gen.convdiff27(16, 15, 17), (16, 15, 17)
    n = A.shape[0]
    rng = np.random.default_rng(7)
    l, r = (rng.integers(-int(1.66 * decades), int(1.66 * decades) + 1, n) for _ in range(2))
    if kind == "rows":
        r = 0 * r
    elif kind == "columns":
        l = 0 * l
    elif kind == "both alike":
        l = r = l // 2
    elif kind == "rows of one half":
        l, r = np.where(np.arange(n) < n // 2, int(3.3 * decades), 0), 0 * r
    xt = gen.rhs_uniform(n, 1, 3)[:, 0]
    ref, flagged = _lu_error(A, grid, A, xt, 0 * l, 0 * r)
    assert flagged == 0
    M = (sps.diags(np.ldexp(1.0, l)) @ A @ sps.diags(np.ldexp(1.0, r))).tocsc()
    err, flagged = _lu_error(M, grid, A, xt, l, r)
    assert err < 2 * ref, (err, ref)
    assert (flagged > 0) == (kind != "both alike")
    assert kind != "rows of one half" or flagged < 1


@pytest.mark.parametrize("kind", ["dropped", "most dropped", "one direction", "lower", "uneven"])
def test_lu_of_unsymmetric_matrices(lib, kind):
    """Unsymmetric patterns, weak couplings in one direction, entries of very different sizes: the slices keep them,
    with the error of FP64 arithmetic (twice that for the order of the scattered sums)."""
    A, grid = gen.convdiff27(24, 23, 25), (24, 23, 25)
    n = A.shape[0]
    rng = np.random.default_rng(11)
    C = A.tocoo()
    off = C.row != C.col
    if kind == "dropped":
        C.data[off & (rng.random(C.nnz) < 0.3)] = 0.0
    elif kind == "most dropped":
        C.data[off & (rng.random(C.nnz) < 0.8)] = 0.0
    elif kind == "one direction":
        C.data[C.row < C.col] *= 1e-8
    elif kind == "lower":
        C.data[C.row < C.col] = 0.0
    else:
        C.data[off] *= 10.0 ** rng.uniform(-8, 0, int(off.sum()))
    A = C.tocsc()
    xt = gen.rhs_uniform(n, 1, 3)[:, 0]
    z = np.zeros(n, dtype=int)
    ref, _ = _lu_error(A, grid, A, xt, z, z, integer=False, min_bs=64, max_bs=128)
    err, flagged = _lu_error(A, grid, A, xt, z, z, min_bs=64, max_bs=128)
    assert err < 2 * ref and flagged == 0, (err, ref, flagged)


def _dense_chain(A, fact, width):
    """Handle of a full matrix cut into panels of `width` columns, in the given order."""
    n = A.shape[0]
    ip, dp = px.initParam()
    ip[px.iparm.factorization] = FACT_ID[fact]
    pd = px.init(ip, dp)
    S = spmatrix(sps.csc_matrix(A), mtxtype.General if fact == "GETRF" else mtxtype.Symmetric)
    rang = np.append(np.arange(0, n, width), n).astype(np.int64)
    tree = np.append(np.arange(1, len(rang) - 1), -1).astype(np.int64)
    px.subtask_order(pd, S, np.arange(n), rang, tree)
    px.subtask_symbfact(pd)
    px.subtask_blend(pd)
    return pd, S, px.solver_info(pd)


def _dense_factor(info, panels):
    """The lower triangle (with the diagonal) held in the panels of a full matrix."""
    n = int(info["cb_lcol"][-1]) + 1
    F = np.zeros((n, n))
    for k in range(int(info["cblknbr"])):
        fc, lc, st, base = (int(info[q][k]) for q in ("cb_fcol", "cb_lcol", "cb_stride", "cb_coef"))
        for c in range(fc, lc + 1):
            F[c:, c] = panels[base + (c - fc) * st + (c - fc): base + (c - fc + 1) * st]
    return F


def _lu(A, width):
    """LU without pivoting in the precision of A, updates in panels of `width` columns (0: column by column)."""
    A, n = A.copy(), len(A)
    w = width or n
    for k in range(0, n, w):
        e = min(n, k + w)
        for c in range(k, e):
            A[c + 1:, c] /= A[c, c]
            A[c + 1:, c + 1:e] -= np.outer(A[c + 1:, c], A[c, c + 1:e])
        for c in range(k, e):
            A[c, e:] -= A[c, k:c] @ A[k:c, e:]
        A[e:, e:] -= A[e:, k:e] @ A[k:e, e:]
    return A


@pytest.mark.parametrize("fact", ["POTRF", "SYTRF", "GETRF"])
@pytest.mark.parametrize("width", [64, 100])
def test_updates_lose_nothing_against_fp64(lib, fact, width):
    """A full matrix whose factor rows hold entries of many sizes that seldom face each other, against its
    elimination in 64-bit mantissas.  Yardstick: the error of the same elimination in FP64; half as much
    again is left for another order of its sums."""
    rng = np.random.default_rng(0)
    n = 520
    q = rng.permutation(n)
    A = np.exp(-np.abs(np.subtract.outer(q, q)) / 20.0) + 0.05 * np.eye(n)
    if fact == "GETRF":
        A *= 1.0 + 0.01 * np.random.default_rng(1).uniform(-1, 1, (n, n))
    ref = _lu(A.astype(np.longdouble), 0)
    e64 = (_lu(A, width) - ref).astype(float)
    pd, S, info = _dense_chain(A, fact, width)
    assert int((info["cb_lcol"] - info["cb_fcol"]).max()) + 1 == width
    px.task_numfact(pd, S)
    Lg, Ug = px.get_coeftab(pd, with_u=(fact == "GETRF"))
    F = _dense_factor(info, Lg)
    d = np.sqrt(np.diag(ref).astype(float))
    if fact == "POTRF":
        got, want = np.tril(F), np.tril(ref, -1) * d[None, :] + np.diag(d)
        e64 = np.tril(e64, -1) * d[None, :]
    else:
        got, want = np.tril(F, -1), np.tril(ref, -1)
        e64 = np.tril(e64, -1)
    err = np.linalg.norm(np.tril((got - want).astype(float), -1))
    assert err < 1.5 * np.linalg.norm(e64)
    if fact == "GETRF":
        Ut = np.tril(_dense_factor(info, Ug), -1)
        e64 = np.triu((_lu(A, width) - ref).astype(float), 1)
        err = np.linalg.norm(Ut - np.triu(ref, 1).T.astype(float))
        assert err < 1.5 * np.linalg.norm(e64)
    px.finalize(pd)


def test_lu_non_finite_entry_reaches_the_solution(lib):
    A, grid = _system("GETRF")
    pd, S, info = analyse(A, grid, "GETRF")
    v = S.values.copy()
    v[A.nnz // 2] = np.inf
    S.set_values(v)
    px.task_numfact(pd, S)
    x = np.ones(A.shape[0])
    px.task_solve(pd, S, x)
    assert np.isnan(x).any()
    px.finalize(pd)


def test_non_finite_entry_reaches_the_solution(lib):
    A, grid = _system("POTRF")
    pd, S, info = analyse(A, grid, "POTRF")
    v = S.values.copy()
    v[0] = np.nan
    S.set_values(v)
    px.task_numfact(pd, S)
    x = np.ones(A.shape[0])
    px.task_solve(pd, S, x)
    assert np.isnan(x).any()
    px.finalize(pd)
