"""FP64 factorizations of 2e10 flops and more run the integer updates of far targets
on a second stream beside the next level's panels: image areas that levels share in
turn, a limited number of tiles per CTA, reductions in place of exclusive writes, LU
sources left to DMMA on the first stream.

Against the same factorization on one stream (per-launch profiling uses one), which
differs in the order of the scattered sums only: an entry is the sum of at most a
few hundred of them, each rounded once, so that 1e3 u = 1e-13 bounds the difference.  The grids give one level at least
more than six tiles for each of 148 CTAs (48^3 Laplacian 990, 36^3 with 27 points
1657), so that CTAs stop at their share."""
from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sps
import torch

from conftest import analyse
from pastix_b200 import gen
from pastix_b200 import pastix as px
from test_gpu_parity import _mask_compare

pytestmark = pytest.mark.gpu


def _factor(pd, vals, fact, keep, one_stream):
    px.profile(pd, one_stream)
    px.numfact_device(pd, vals)
    L, U = px.get_coeftab(pd, with_u=(fact == "GETRF"))
    launches = px.profile_get(pd)["update_big"][1]
    px.profile(pd, False)
    return [L[keep]] + ([U] if U is not None else []), launches


@pytest.mark.parametrize("fact,uneven", [("POTRF", False), ("SYTRF", False), ("GETRF", False), ("GETRF", True)])
def test_two_streams_give_the_factors_of_one(lib, fact, uneven):
    grid = (36, 36, 36) if fact == "GETRF" else (48, 48, 48)
    A = gen.convdiff27(*grid) if fact == "GETRF" else gen.laplacian7(*grid)
    rng = np.random.default_rng(5)
    if uneven:  # rows of a part of the domain in other units: some sources are left to DMMA
        A = (sps.diags(np.where(np.arange(A.shape[0]) < A.shape[0] // 8, 2.0 ** 20, 1.0)) @ A).tocsc()
    pd, S, info = analyse(A, grid, fact)
    assert info["thflops"] >= 2e10
    keep = _mask_compare(fact, info)
    # new values for every pass: nothing of the one before may be left in the images
    vals = [torch.tensor(S.values * s, device="cuda") for s in (1.0, 3.0)]
    for v in vals:
        one, n1 = _factor(pd, v, fact, keep, True)
        flagged = px.get_update_path(pd)[1]
        for _ in range(2):
            two, n2 = _factor(pd, v, fact, keep, False)
            assert n2 > n1  # near and far targets in launches of their own
            used, fl = px.get_update_path(pd)
            assert used and fl == flagged and (flagged > 0) == uneven
            for a, b in zip(two, one):
                assert np.linalg.norm(a - b) / np.linalg.norm(b) < 1e-13
    assert lib.pgpu_device_status(pd.ptr) == 0
    xt = rng.uniform(-1, 1, S.n)
    x = torch.tensor(3.0 * (S.full() @ xt), device="cuda")
    px.solve_device(pd, x)
    assert np.linalg.norm(x.cpu().numpy() - xt) / np.linalg.norm(xt) < 1e-11
    px.finalize(pd)
