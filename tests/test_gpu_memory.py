"""Device memory of the FP64 factorization's digit images: they are taken only with
room to spare, and are given back when a solve finds no other memory.

The device is filled by one allocation down to a stated rest; every failure is an
allocation that returns an error."""
from __future__ import annotations

import contextlib

import numpy as np
import pytest
import torch

from conftest import analyse
from pastix_b200 import gen
from pastix_b200 import pastix as px

pytestmark = pytest.mark.gpu

MIB = 1 << 20


@contextlib.contextmanager
def _filled(rest):
    """One allocation that leaves about `rest` bytes of the device free."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    hog = torch.empty(max(1, torch.cuda.mem_get_info()[0] - rest), dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del hog
        torch.cuda.empty_cache()


def _handle(fact):
    A = gen.convdiff27(18, 18, 18) if fact == "GETRF" else gen.laplacian7(30, 30, 30)
    grid = (18, 18, 18) if fact == "GETRF" else (30, 30, 30)
    pd, S, info = analyse(A, grid, fact)
    return pd, S, torch.tensor(S.values, device="cuda")


def _solves(pd, S, nrhs=1):
    xt = np.random.default_rng(2).uniform(-1, 1, (S.n, nrhs))
    x = torch.tensor(np.ascontiguousarray((S.full() @ xt).T), device="cuda").t()
    px.solve_device(pd, x)
    return np.linalg.norm(x.cpu().numpy() - xt) / np.linalg.norm(xt) < 1e-12


@pytest.mark.parametrize("fact", ["POTRF", "SYTRF", "GETRF"])
def test_images_leave_room(lib, fact):
    pd, S, v = _handle(fact)
    px.integer_updates(pd, False)
    px.numfact_device(pd, v)
    px.integer_updates(pd, True)
    with _filled(300 * MIB):  # holds the images, but not what is left free beside them
        px.numfact_device(pd, v)
        assert px.get_update_path(pd) == (False, 0)
        assert _solves(pd, S)
    px.numfact_device(pd, v)
    assert px.get_update_path(pd) == (False, 0)  # not tried again on every call
    px.integer_updates(pd, True)
    px.numfact_device(pd, v)
    assert px.get_update_path(pd) == (True, 0)
    assert _solves(pd, S)
    px.finalize(pd)


@pytest.mark.parametrize("fact", ["POTRF", "GETRF"])
def test_images_are_given_back(lib, fact):
    pd, S, v = _handle(fact)
    px.integer_updates(pd, False)
    px.numfact_device(pd, v)
    assert _solves(pd, S)  # work vectors and graphs in place
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    px.integer_updates(pd, True)
    px.numfact_device(pd, v)
    images = before - torch.cuda.mem_get_info()[0]
    assert images >= 8 * MIB and px.get_update_path(pd) == (True, 0)
    rest = images // 2
    nrhs = (rest + images // 4) // (8 * S.n)  # its work vectors need more than is free, less than with the images
    xt = np.random.default_rng(2).uniform(-1, 1, (S.n, nrhs))
    x = torch.tensor(np.ascontiguousarray((S.full() @ xt).T), device="cuda").t()
    with _filled(rest):
        px.solve_device(pd, x)
    assert np.linalg.norm(x.cpu().numpy() - xt) / np.linalg.norm(xt) < 1e-12
    px.numfact_device(pd, v)
    assert px.get_update_path(pd) == (False, 0)
    assert _solves(pd, S, 3)
    px.finalize(pd)


def test_failed_factorization_leaves_the_values_in_place(lib):
    """Panels that cannot be allocated: the call fails after the values were taken.  They and their norm are complete
    when it returns, and a product on another stream sees them."""
    pd, S, v = _handle("POTRF")
    pd.iparm[px.iparm.mixed] = 1
    px.numfact_device(pd, v)
    pd.iparm[px.iparm.mixed] = 0  # panels of twice the size
    w = 2.0 * v
    pd.dparm[px.dparm.a_norm] = 0.0
    with _filled(8 * MIB), pytest.raises(px.PastixError):
        px.numfact_device(pd, w)
    norm = float(pd.dparm[px.dparm.a_norm])
    A = 2.0 * S.full()
    assert abs(norm - np.sqrt((A.data ** 2).sum())) < 1e-12 * norm
    x = torch.rand(S.n, dtype=torch.float64, device="cuda")
    y = torch.zeros_like(x)
    px.spmv_device(pd, 1.0, x, 0.0, y)
    assert np.linalg.norm(y.cpu().numpy() - A @ x.cpu().numpy()) < 1e-13 * np.linalg.norm(y.cpu().numpy())
    px.numfact_device(pd, w)
    assert px.get_update_path(pd) == (True, 0)
    px.finalize(pd)
