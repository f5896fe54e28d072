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

from conftest import analyse, backward_error
from pastix_b200 import gen
from pastix_b200 import pastix as px
from test_gpu_parity import _mask_compare

pytestmark = pytest.mark.gpu


def _system(fact):
    if fact == "GETRF":
        return gen.convdiff27(15, 14, 13), (15, 14, 13)
    return gen.laplacian7(17, 18, 19), (17, 18, 19)


@pytest.mark.parametrize("fact", ["POTRF", "SYTRF", "GETRF"])
@pytest.mark.parametrize("bs", [(32, 33), (40, 64), (64, 65), (96, 129), (160, 320)])
def test_factors_at_tile_edges(lib, oracle_mod, fact, bs):
    A, grid = _system(fact)
    pd, S, info = analyse(A, grid, fact, min_bs=bs[0], max_bs=bs[1])
    px.task_numfact(pd, S)
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
