"""SpMV in the caller's numbering against the oracle's product, and with x and y
in the same memory (the copy path): y = alpha A x + beta x."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import analyse
from pastix_b200 import gen
from pastix_b200 import pastix as px

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beta", [0.0, -0.75])
@pytest.mark.parametrize("shift", [None, 0, 3])
def test_spmv_overlap(lib, beta, shift):
    torch = pytest.importorskip("torch")
    A = gen.convdiff27(9, 8, 7)
    n = A.shape[0]
    pd, S, _ = analyse(A, (9, 8, 7), "GETRF")
    px.task_numfact(pd, S)
    buf = torch.tensor(np.random.default_rng(1).standard_normal(2 * n + 8), device="cuda")
    x, y = buf[:n], (buf[n + 8:] if shift is None else buf[shift:shift + n])
    ref = 1.5 * (S.full() @ x.cpu().numpy()) + beta * y.cpu().numpy()
    px.spmv_device(pd, 1.5, x, beta, y)
    # sums of at most 27 products: 28 u relative to the sum of magnitudes
    assert np.abs(y.cpu().numpy() - ref).max() <= 28 * 2.0 ** -52 * np.abs(ref).max() * 8
    px.finalize(pd)
