"""Off-diagonal triangular solves of the FP64 factorization at the edges of their
tiles: blocks of 33 to 484 columns, and panels whose numbers of rows leave
partial tiles and unpaired ones, in levels with few and with many tiles.  The
LU case of 306 columns takes the 16-CTA clusters of the diagonal blocks.

Factors against the oracle's, entry sums of at most n products: n u = 6e-13.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import analyse
from pastix_b200 import gen
from pastix_b200 import pastix as px
from test_gpu_parity import _mask_compare

pytestmark = pytest.mark.gpu


SMALL = [((13, 13, 20), (33, 34)), ((9, 10, 40), (80, 90)), ((40, 31, 3), (40, 64))]
CASES = [(f, g, b) for f in ("POTRF", "SYTRF", "GETRF") for g, b in SMALL]
CASES += [("POTRF", (21, 22, 23), (300, 384)), ("GETRF", (18, 17, 19), (300, 330)), ("SYTRF", (18, 18, 18), (320, 330))]


@pytest.mark.parametrize("fact,grid,bs", CASES)
def test_factor_edges(lib, oracle_mod, fact, grid, bs):
    A = gen.convdiff27(*grid) if fact == "GETRF" else gen.laplacian7(*grid)
    pd, S, info = analyse(A, grid, fact, min_bs=bs[0], max_bs=bs[1])
    px.task_numfact(pd, S)
    Lg, Ug = px.get_coeftab(pd, with_u=(fact == "GETRF"))
    sym = oracle_mod.Symbol(info)
    Ap = oracle_mod.permuted_full(S.full(), info["permtab"])
    L2, U2, npiv = oracle_mod.factor(sym, Ap, fact, oracle_mod.criterion(Ap))
    assert int(pd.iparm[px.iparm.static_pivoting]) == npiv
    keep = _mask_compare(fact, info)
    Lo = oracle_mod.to_panels(sym, L2)
    assert np.linalg.norm((Lg - Lo)[keep]) / np.linalg.norm(Lo[keep]) < 6e-13
    if fact == "GETRF":
        Uo = oracle_mod.to_panels(sym, U2)
        assert np.linalg.norm(Ug - Uo) / np.linalg.norm(Uo) < 6e-13
    px.finalize(pd)
