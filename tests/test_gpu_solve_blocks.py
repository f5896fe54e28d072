"""Solve kernels at the edges of their blocks: cblk widths around the 32-column
steps of the diagonal solves and the 64 x 64 tiles of the off-diagonal updates
(up to 484 columns: the supernode that IPARM_MIN_BLOCKSIZE leaves whole), and numbers of right-hand sides around the groups of 8.

The bar is the backward error of a stable solve: the sums have at most a few
thousand terms, so n u = 2e-13 bounds it in FP64 (observed 1e-16); FP32 factors
are compared at their own roundoff, n 2^-24 = 1e-4 (observed 1e-7).
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import analyse, backward_error
from pastix_b200 import gen
from pastix_b200 import pastix as px

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fact", ["POTRF", "SYTRF", "GETRF"])
@pytest.mark.parametrize("bs", [(32, 33), (63, 64), (64, 65), (95, 97), (300, 384)])
@pytest.mark.parametrize("mixed", [False, True])
def test_solve_block_edges(lib, fact, bs, mixed):
    torch = pytest.importorskip("torch")
    A = gen.convdiff27(16, 15, 13) if fact == "GETRF" else gen.laplacian7(21, 22, 23)
    grid = (16, 15, 13) if fact == "GETRF" else (21, 22, 23)
    pd, S, info = analyse(A, grid, fact, mixed=mixed, min_bs=bs[0], max_bs=bs[1])
    px.task_numfact(pd, S)
    assert bs[1] < 384 or fact == "GETRF" or int((info["cb_lcol"] - info["cb_fcol"]).max()) + 1 > 384
    Af = S.full()
    for nrhs in (1, 2, 7, 8, 9, 17, 33):
        b = np.asfortranarray(Af @ gen.rhs_uniform(A.shape[0], nrhs, nrhs))
        for trans in (False, True) if fact == "GETRF" else (False,):
            x = torch.from_numpy(np.ascontiguousarray(b.T)).cuda().t()
            px.solve_device(pd, x, transposed=trans)
            xh = x.cpu().numpy()
            M = Af.T if trans else Af
            for j in range(nrhs):
                assert backward_error(M, xh[:, j], b[:, j]) < (1e-4 if mixed else 2e-13), (nrhs, j)
    px.finalize(pd)
