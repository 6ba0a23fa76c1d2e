"""GPU: kernels at the sizes where their tiles, remainders and dispatch rules can go wrong,
against the oracle.  Tolerances: a sum of n terms of one sign carries at most about
n * 1.1e-16 relative error (n <= 1000 taps: 1e-13)."""
import ctypes

import numpy as np
import pytest
import torch

from conftest import rel
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    from pyfantom_b200 import _lib
    _lib.require_cuda()
    return _lib


def T(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device="cuda")


def N(t):
    torch.cuda.synchronize()
    return t.detach().cpu().numpy()


@pytest.mark.parametrize("nel,r,h", [
    ((1, 1, 1), 2.0, (1, 1, 1)), ((3, 2, 5), 3.5, (1, 1, 1)), ((9, 16, 32), 2.0, (1, 1, 1)),
    ((17, 15, 33), 2.5, (1, 1, 1)), ((64, 48, 48), 2.0, (1, 1, 1)), ((95, 47, 49), 1.5, (1, 1, 1)),
    ((130, 66, 67), 2.5, (1, 1, 1)), ((20, 18, 24), 4.2, (1, 1, 1)), ((21, 19, 34), 5.0, (1, 1, 1)),
    ((18, 17, 40), 6.0, (1, 1, 1)), ((24, 20, 16), 2.5, (1.0, 1.25, 2.0)), ((120, 40), 1.5, (1, 1)), ((33, 257), 3.0, (1, 1)),
    ((7, 8), 12.0, (1, 1))])
def test_filter_tiles(lib, nel, r, h):
    w, off = O.filter_weights(nel, h, r)
    grid, f = lib.make_grid(nel), ctypes.c_void_p()
    L = lib.load()
    off = np.ascontiguousarray(off, dtype=np.int32)
    w = np.ascontiguousarray(w)
    lib.check(L.pf_filter_create(ctypes.byref(grid), len(w), off.ctypes.data, w.ctypes.data, ctypes.byref(f)))
    v = np.random.default_rng(3).uniform(0.1, 1.0, int(np.prod(nel)))
    vt = T(v)
    y, z = torch.full_like(vt, np.nan), torch.full_like(vt, np.nan)
    lib.check(L.pf_filter_fwd_f64(f, lib.ptr(vt), lib.ptr(y), lib.stream()))
    lib.check(L.pf_filter_adj_f64(f, lib.ptr(vt), lib.ptr(z), lib.stream()))
    assert rel(N(y), O.filter_fwd(nel, w, off, v)) < 1e-13
    assert rel(N(z), O.filter_adj(nel, w, off, O.filter_normalizer(nel, w, off), v)) < 1e-13
    L.pf_filter_destroy(f)


def test_filter_taps_that_are_no_columns(lib):
    # an offset set with a hole along x: served by the general kernel
    nel = (12, 9, 10)
    off = np.array([[-2, 0, 0], [0, 0, 0], [2, 0, 0], [0, 1, 0], [0, -1, 0]], dtype=np.int32)
    w = np.array([0.2, 0.3, 0.2, 0.15, 0.15])
    grid, f = lib.make_grid(nel), ctypes.c_void_p()
    L = lib.load()
    lib.check(L.pf_filter_create(ctypes.byref(grid), len(w), off.ctypes.data, w.ctypes.data, ctypes.byref(f)))
    v = np.random.default_rng(4).uniform(0.1, 1.0, int(np.prod(nel)))
    vt = T(v)
    y = torch.empty_like(vt)
    lib.check(L.pf_filter_fwd_f64(f, lib.ptr(vt), lib.ptr(y), lib.stream()))
    assert rel(N(y), O.filter_fwd(nel, w, off, v)) < 1e-13
    L.pf_filter_destroy(f)
