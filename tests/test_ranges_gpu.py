"""GPU: kernels at the sizes where their tiles, remainders and dispatch rules can go wrong,
against the oracle.  Tolerances: a sum of n terms of one sign carries at most about
n * 1.1e-16 relative error (n <= 1000 taps: 1e-13)."""
import ctypes
from fractions import Fraction

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


def _oc(lib, x, df, dg, vf, move, wait=True):
    L = lib.load()
    n = len(x)
    xt, ft, gt = T(x), T(df), T(dg)
    work = torch.full((int(L.pf_oc_workspace_size(n)),), np.nan, dtype=torch.float64, device="cuda")
    xn = torch.full_like(xt, np.nan)
    out = (ctypes.c_double * 3)()
    lib.check(L.pf_oc_update_f64(n, lib.ptr(xt), lib.ptr(ft), lib.ptr(gt), vf, move, lib.ptr(xn), lib.ptr(work),
                                 out if wait else None, lib.stream()))
    return N(xn), list(out)


@pytest.mark.parametrize("n", [1, 31, 255, 257, 4800, 75_777, 300_001])
@pytest.mark.parametrize("kind", ["usual", "tiny", "huge", "slack", "tight", "zero", "signs", "flat"])
def test_oc_sequences(lib, n, kind):
    # multipliers over the whole bracket, volumes met everywhere or nowhere, a zero gradient,
    # a constraint gradient of both signs (no falling volume: five levels a pass from the start)
    rng = np.random.default_rng(n)
    x = rng.uniform(0.05, 0.95, n)
    df = -np.exp(rng.normal(0.0, 2.0, n))
    dg = rng.uniform(0.5, 1.5, n) / n
    vf, move = 0.4 * dg.sum(), 0.2
    if kind == "tiny":
        df = df * 1e-18 / n
    elif kind == "huge":
        df = df * 1e14
    elif kind == "slack":
        vf = 2.0
    elif kind == "tight":
        vf = -1.0
    elif kind == "zero":
        df = np.abs(df)
    elif kind == "signs":
        dg = np.where(rng.uniform(size=n) < 0.2, -dg, dg)
    elif kind == "flat":
        x, df, dg = np.full(n, 0.4), np.full(n, -1.0), np.full(n, 1.0 / n)
    ref, steps = O.oc_update(x, df, dg, vf, move)
    got, out = _oc(lib, x, df, dg, vf, move)
    assert int(out[2]) == steps
    # the sums differ in order only: the bisection ends within its own tolerance of 1e-8, and
    # takes another branch only where the volume is met to 1e-13
    assert np.abs(got - ref).max() < 1e-9 or kind == "flat"
    if kind == "flat":  # every element at the volume fraction itself: the last steps are ties
        assert np.abs(got - ref).max() < 2e-8
    late, _ = _oc(lib, x, df, dg, vf, move, wait=False)
    assert np.array_equal(late, got)


@pytest.mark.parametrize("n", [257, 4800, 300_001])
@pytest.mark.parametrize("where", ["x", "df", "dg", "dg+1", "dg-3"])
@pytest.mark.parametrize("entry", ["work", "noalloc"])
def test_oc_result_over_an_operand(lib, n, where, entry):
    # x_new in the memory of an operand; the bounds are those of the separate buffers above
    rng = np.random.default_rng(n)
    x, df = rng.uniform(0.05, 0.95, n), -np.exp(rng.normal(0.0, 2.0, n))
    dg = rng.uniform(0.5, 1.5, n) / n
    vf, move = 0.4 * dg.sum(), 0.2
    ref, steps = O.oc_update(x, df, dg, vf, move)
    big = torch.full((n + 8,), np.nan, dtype=torch.float64, device="cuda")
    big[4:n + 4] = T(dg)
    xt, ft, gt = T(x), T(df), big[4:n + 4]
    xn = {"x": xt, "df": ft, "dg": gt, "dg+1": big[5:n + 5], "dg-3": big[1:n + 1]}[where]
    L = lib.load()
    out = (ctypes.c_double * 3)()
    if entry == "work":
        work = torch.empty(int(L.pf_oc_workspace_size(n)), dtype=torch.float64, device="cuda")
        lib.check(L.pf_oc_update_f64(n, lib.ptr(xt), lib.ptr(ft), lib.ptr(gt), vf, move, lib.ptr(xn), lib.ptr(work), out,
                                     lib.stream()))
    else:
        lib.check(L.pf_oc_update_noalloc_f64(n, lib.ptr(xt), lib.ptr(ft), lib.ptr(gt), vf, move, lib.ptr(xn), out,
                                             lib.stream()))
    assert int(out[2]) == steps
    assert np.abs(N(xn) - ref).max() < 1e-9


@pytest.mark.parametrize("shape,co,stride", [
    ((1, 1, 1, 1, 1), 1, 1), ((1, 17, 2, 16, 8), 17, 1), ((2, 57, 5, 17, 9), 65, 1), ((1, 64, 3, 33, 17), 48, 2),
    ((2, 16, 16, 32, 32), 16, 1), ((8, 8, 32, 16, 16), 16, 1), ((1, 130, 4, 5, 20), 130, 1), ((1, 33, 1, 2, 3), 20, 2),
    ((3, 16, 18, 20, 34), 32, 2)])
def test_conv_tiles(lib, shape, co, stride):
    # tile edges along each axis, channel chunks of 16 with a remainder, column splits, several
    # input-channel tiles; operands representable in BF16, so only the FP32 accumulation differs
    # from float64 (sums of up to 27 * 130 products or 12,000 voxels: 1e-5 of the largest entry)
    N_, ci, X, Y, Z = shape
    g = torch.Generator(device="cuda").manual_seed(7)
    def bf(*s):
        return torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16).to(torch.float32)
    x, w, b = bf(*shape), bf(co, ci, 3, 3, 3), torch.randn(co, generator=g, device="cuda")
    xd, wd = x.double().requires_grad_(), w.double().requires_grad_()
    ref = torch.nn.functional.conv3d(xd, wd, b.double(), stride=stride, padding=1)
    dy = bf(*ref.shape)
    gx, gw = torch.autograd.grad(ref, (xd, wd), dy.double())
    L = lib.load()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    y, dx = torch.full_like(dy, np.nan), torch.full_like(x, np.nan)
    dw, db = torch.full_like(w, np.nan), torch.full_like(b, np.nan)
    nw = int(L.pf_cnn_conv3d_bwd_weight_tc_workspace(N_, ci, X, Y, Z, co, stride))
    work = torch.full((nw,), np.nan, dtype=torch.float32, device="cuda")
    P = lib.ptr
    lib.check(L.pf_cnn_conv3d_fwd_tc(P(x), N_, ci, X, Y, Z, P(w), P(b), co, stride, 0, P(y), P(err), lib.stream()))
    lib.check(L.pf_cnn_conv3d_bwd_data_tc(P(dy), N_, ci, X, Y, Z, P(w), co, stride, 0, P(dx), P(err), lib.stream()))
    lib.check(L.pf_cnn_conv3d_bwd_weight_tc(P(x), P(dy), N_, ci, X, Y, Z, co, stride, P(dw), P(db), P(work), P(err),
                                            lib.stream()))
    assert int(err.item()) == 0
    for got, want in ((y, ref), (dx, gx), (dw, gw), (db, dy.double().sum(dim=(0, 2, 3, 4)))):
        assert rel(N(got), N(want)) < 1e-5


@pytest.mark.parametrize("ci,co,stride", [(1, 240, 1), (200, 2, 1), (130, 1, 2)])
def test_conv_of_many_samples(lib, ci, co, stride):
    # samples times column splits beyond 65,535 (three or four splits of the output or input channels)
    n, ext = 22_000 if max(ci, co) < 150 else 17_000, (2, 1, 1)
    L, P, s = lib.load(), lib.ptr, lib.stream()
    g = torch.Generator(device="cuda").manual_seed(9)
    w, b = torch.randn(co, ci, 3, 3, 3, generator=g, device="cuda").bfloat16().float(), torch.zeros(co, device="cuda")
    x = torch.randn(n, ci, *ext, generator=g, device="cuda").bfloat16().float()
    xd, wd = x.double().requires_grad_(), w.double()
    xp = torch.nn.functional.pad(xd[:, :, :, 0, 0], (1, 1))
    outs = [torch.einsum("nit,oit->no", xp[:, :, stride * o:stride * o + 3], wd[:, :, :, 1, 1]) for o in range(2 // stride)]
    ref = torch.stack(outs, 2)[..., None, None]
    dy = torch.randn(ref.shape, generator=g, device="cuda").bfloat16().float()
    gx, = torch.autograd.grad(ref, xd, dy.double())
    y, dx = torch.full_like(dy, np.nan), torch.full_like(x, np.nan)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    lib.check(L.pf_cnn_conv3d_fwd_tc(P(x), n, ci, *ext, P(w), P(b), co, stride, 0, P(y), P(err), s))
    lib.check(L.pf_cnn_conv3d_bwd_data_tc(P(dy), n, ci, *ext, P(w), co, stride, 0, P(dx), P(err), s))
    assert int(err.item()) == 0
    # operands representable in BF16: only the FP32 accumulation differs, as in test_conv_tiles
    assert rel(N(y), N(ref)) < 1e-5 and rel(N(dx), N(gx)) < 1e-5


@pytest.mark.parametrize("stride", [1, 2])
def test_conv_beyond_32_bit_offsets(lib, stride):
    # one channel of more than 2^31 voxels, zero but for its last planes: results there as those of a grid that
    # holds the last planes alone (cut where tiles begin), bitwise for the same products and sums
    X, Y, Z, tail = 2080, 1024, 1024, 32
    L, P, s = lib.load(), lib.ptr, lib.stream()
    g = torch.Generator(device="cuda").manual_seed(5)
    w, b = torch.randn(1, 1, 3, 3, 3, generator=g, device="cuda"), torch.randn(1, generator=g, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    x = torch.zeros(X, Y, Z, device="cuda")
    x[X - tail + 1:] = torch.randn(tail - 1, Y, Z, generator=g, device="cuda")
    so = [(v - 1) // stride + 1 for v in (X, Y, Z)]
    dy = torch.zeros(so, device="cuda")
    ot = tail // stride  # output planes of the last ones; the first of them stays zero
    dy[so[0] - ot + 1:] = torch.randn(ot - 1, *so[1:], generator=g, device="cuda")

    def passes(x, dy):
        n = (1, 1, *x.shape)
        y, dx, dw, db = torch.empty_like(dy), torch.empty_like(x), torch.empty_like(w), torch.empty_like(b)
        lib.check(L.pf_cnn_conv3d_fwd_tc(P(x), *n, P(w), P(b), 1, stride, 0, P(y), P(err), s))
        lib.check(L.pf_cnn_conv3d_bwd_data_tc(P(dy), *n, P(w), 1, stride, 0, P(dx), P(err), s))
        work = torch.empty(int(L.pf_cnn_conv3d_bwd_weight_tc_workspace(*n, 1, stride)), device="cuda")
        lib.check(L.pf_cnn_conv3d_bwd_weight_tc(P(x), P(dy), *n, 1, stride, P(dw), P(db), P(work), P(err), s))
        return y, dx, dw, db

    y, dx, dw, db = passes(x, dy)
    y1, dx1, dw1, db1 = passes(x[X - tail:].contiguous(), dy[so[0] - ot:].contiguous())
    assert int(err.item()) == 0
    assert torch.equal(y[so[0] - ot:], y1) and torch.equal(dx[X - tail:], dx1)
    assert bool((y[:so[0] - ot - 1] == b).all()) and bool((dx[:X - tail - 1] == 0).all())
    # the weight gradient's ranges lie elsewhere: sums of up to 33 million products in FP32, by ranges of 4096
    assert rel(N(dw), N(dw1)) < 1e-4 and rel(N(db), N(db1)) < 1e-4


@pytest.mark.parametrize("ext,stride", [((5, 17, 9), 1), ((4, 16, 8), 1), ((3, 5, 3), 1), ((6, 18, 10), 2), ((7, 35, 21), 2),
                                       ((2, 33, 20), 1)])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_conv_weight_gradient_of_infinities(lib, ext, stride, bad):
    # one infinity or NaN per channel on an upper face, an edge, a corner, inside: exactly the taps that meet it
    # with a valid output are not finite; the others as in test_conv_tiles
    N_, ci, co = 2, 9, 17
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(N_, ci, *ext, generator=g, device="cuda").to(torch.bfloat16).to(torch.float32)
    hi, mid = [v - 1 for v in ext], [v // 2 for v in ext]
    for c, at in enumerate([(hi[0], mid[1], mid[2]), (mid[0], hi[1], mid[2]), (mid[0], mid[1], hi[2]), (hi[0], hi[1], mid[2]),
                            (mid[0], hi[1], hi[2]), tuple(hi), tuple(mid)]):
        x[1, c, at[0], at[1], at[2]] = bad
    outs = [(v - 1) // stride + 1 for v in ext]
    dy = torch.randn(N_, co, *outs, generator=g, device="cuda").to(torch.bfloat16).to(torch.float32)
    xp = torch.nn.functional.pad(x.double(), (1,) * 6)
    ref = torch.empty(co, ci, 3, 3, 3, dtype=torch.float64, device="cuda")
    for t in range(27):
        o = (t // 9, t // 3 % 3, t % 3)
        xs = xp[(slice(None), slice(None), *(slice(o[a], o[a] + stride * (outs[a] - 1) + 1, stride) for a in range(3)))]
        ref[:, :, o[0], o[1], o[2]] = (xs[:, None] * dy.double()[:, :, None]).sum(dim=(0, 3, 4, 5))
    L, P = lib.load(), lib.ptr
    dw, db = torch.zeros(co, ci, 3, 3, 3, device="cuda"), torch.zeros(co, device="cuda")
    work = torch.empty(int(L.pf_cnn_conv3d_bwd_weight_tc_workspace(N_, ci, *ext, co, stride)), device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    lib.check(L.pf_cnn_conv3d_bwd_weight_tc(P(x), P(dy), N_, ci, *ext, co, stride, P(dw), P(db), P(work), P(err), lib.stream()))
    got, want = N(dw), N(ref)
    assert int(err.item()) == 0
    ok = np.isfinite(want)
    assert np.array_equal(ok, np.isfinite(got)) and 0 < ok.sum() < ok.size
    assert np.array_equal(want[~ok], got[~ok].astype(np.float64), equal_nan=True)
    assert np.abs(got[ok] - want[ok]).max() < 1e-5 * np.abs(want[ok]).max()
    assert rel(N(db), N(dy.double().sum(dim=(0, 2, 3, 4)))) < 1e-5


@pytest.mark.parametrize("nel", [(1, 1), (3, 2), (2, 9), (60, 20), (20, 60), (33, 45), (45, 45), (120, 40), (300, 5), (46, 46),
                                 (1, 1, 1), (20, 1, 1), (2, 9, 2), (3, 3, 30), (4, 3, 3), (6, 5, 5)])
def test_direct_band(lib, nel):
    # banded and dense route, either axis the longest, windows and halves of every small size.
    # Cholesky's backward error is a small multiple of (band width) * eps of |K| |x|: 1e-13
    from conftest import unit_K0
    dim = len(nel)
    K0 = unit_K0(dim)
    rng = np.random.default_rng(sum(nel))
    ndof = O.n_nodes(nel) * dim
    E = rng.uniform(0.05, 1.0, O.n_elem(nel))
    # the nodes of the x = 0 face, and a few single DOFs
    nx = nel[0] + 1
    node = np.arange(O.n_nodes(nel))
    ix = (node // (nel[2] + 1 if dim == 3 else 1)) % nx
    cons = np.unique(np.concatenate([(node[ix == 0][:, None] * dim + np.arange(dim)).reshape(-1),
                                     rng.integers(0, ndof, 3)]))
    b = rng.standard_normal(ndof)
    free = np.setdiff1d(np.arange(ndof), cons).astype(np.int32)
    d2f = np.full(ndof, -1, dtype=np.int32)
    d2f[free] = np.arange(len(free), dtype=np.int32)
    L = lib.load()
    grid, op, d = lib.make_grid(nel), ctypes.c_void_p(), ctypes.c_void_p()
    K0c = np.ascontiguousarray(K0)
    lib.check(L.pf_op_create(ctypes.byref(grid), K0c.ctypes.data, ctypes.byref(op)))
    lib.check(L.pf_direct_create(op, ctypes.byref(d)))
    Et, ft, dt, bt = T(E), T(free, torch.int32), T(d2f, torch.int32), T(b)
    x = torch.full_like(bt, np.nan)
    for _ in range(2):
        lib.check(L.pf_direct_solve_f64(d, lib.ptr(Et), lib.ptr(ft), lib.ptr(dt), len(free), lib.ptr(bt), lib.ptr(x),
                                        lib.stream()))
    xs = N(x)
    assert np.array_equal(xs[cons], b[cons])
    u = xs.copy()
    u[cons] = 0.0
    r = (O.matvec(nel, K0, E, u) - b)[free]
    norm = 2 ** dim * np.abs(K0).sum(axis=1).max()
    assert np.linalg.norm(r) < 1e-13 * (norm * np.linalg.norm(u) + np.linalg.norm(b))
    # a stiffness that is not positive definite is reported
    Et[: len(E) // 2 + 1] = -1.0
    assert L.pf_direct_solve_f64(d, lib.ptr(Et), lib.ptr(ft), lib.ptr(dt), len(free), lib.ptr(bt), lib.ptr(x),
                                 lib.stream()) == lib.PF_FACTOR_FAILED
    L.pf_direct_destroy(d)
    L.pf_op_destroy(op)


@pytest.mark.parametrize("nel", [(60, 20), (80, 10), (20, 45), (24, 8), (2, 1), (30, 3, 3), (4, 3, 12)])
def test_direct_band_error(lib, nel):
    # against the exact solution (residuals in integers): the first solve is off by cond(K) (below 1e7) times a few 1e-16,
    # below 1e-9; the correction leaves its square and a few roundings of the result
    from conftest import unit_K0
    dim, K0 = len(nel), unit_K0(len(nel))
    nn = [v + 1 for v in nel]
    ndof = int(np.prod(nn)) * dim
    rng = np.random.default_rng(7)
    E = rng.uniform(0.05, 1.0, int(np.prod(nel)))
    at = np.stack([v.reshape(-1) for v in np.meshgrid(*[np.arange(v) for v in nel], indexing="ij")], 1)
    corners = np.array([(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)])[:2 ** dim, :dim]
    q = at[:, None] + corners
    node = q[..., 0] + nn[0] * q[..., 1] if dim == 2 else q[..., 2] + nn[2] * (q[..., 0] + nn[0] * q[..., 1])
    dofs = (node[..., None] * dim + np.arange(dim)).reshape(len(E), -1)
    ix = (np.arange(ndof) // dim // (nn[2] if dim == 3 else 1)) % nn[0]
    cons = np.nonzero(ix == 0)[0]
    free = np.nonzero(ix != 0)[0].astype(np.int32)
    b = np.zeros(ndof)
    b[ix == nel[0]] = -1.0
    A = np.zeros((ndof, ndof))
    np.add.at(A, (dofs[:, :, None], dofs[:, None, :]), E[:, None, None] * K0)
    inv = np.linalg.inv(A[np.ix_(free, free)])
    fix = np.vectorize(lambda v, bits: int(Fraction(float(v)) * 2 ** bits), otypes=[object])  # exact: no bit is cut off
    Ke = fix(E, 70)[:, None, None] * fix(K0, 130)
    assert np.all(Ke.astype(np.float64) * 2.0 ** -200 == E[:, None, None] * K0)
    x100, b300 = np.zeros(ndof, dtype=object), fix(b, 300)  # x in units of 2^-100
    for _ in range(12):
        y = np.zeros(ndof, dtype=object)
        np.add.at(y, dofs, (Ke * x100[dofs][:, None, :]).sum(axis=-1))
        step = inv @ ((b300 - y)[free].astype(np.float64) * 2.0 ** -300)
        x100[free] += fix(step, 100)
    ref = x100.astype(np.float64) * 2.0 ** -100
    assert np.abs(step).max() < 1e-20 * np.abs(ref).max()
    d2f = np.full(ndof, -1, dtype=np.int32)
    d2f[free] = np.arange(len(free), dtype=np.int32)
    L = lib.load()
    grid, op, d = lib.make_grid(nel), ctypes.c_void_p(), ctypes.c_void_p()
    K0c = np.ascontiguousarray(K0)
    lib.check(L.pf_op_create(ctypes.byref(grid), K0c.ctypes.data, ctypes.byref(op)))
    lib.check(L.pf_direct_create(op, ctypes.byref(d)))
    Et, ft, dt, x = T(E), T(free, torch.int32), T(d2f, torch.int32), T(b)
    lib.check(L.pf_direct_solve_f64(d, lib.ptr(Et), lib.ptr(ft), lib.ptr(dt), len(free), lib.ptr(x), lib.ptr(x), lib.stream()))
    assert float(np.abs((N(x) - ref)[free]).max() / np.abs(ref).max()) < 1e-15
    assert np.array_equal(N(x)[cons], b[cons])
    L.pf_direct_destroy(d)
    L.pf_op_destroy(op)


@pytest.mark.parametrize("nel", [(1, 1, 1), (2, 3, 31), (17, 2, 32), (33, 5, 33), (16, 9, 64), (50, 20, 70)])
def test_sensitivity_march(lib, nel):
    # z remainders of the 32-wide march and chunk ends along x; 24-term quadratic forms: 1e-13
    from conftest import unit_K0
    K0 = np.ascontiguousarray(unit_K0(3, h=(1.0, 1.25, 0.8)))
    U = np.random.default_rng(5).standard_normal(O.n_nodes(nel) * 3)
    L = lib.load()
    grid, op = lib.make_grid(nel), ctypes.c_void_p()
    lib.check(L.pf_op_create(ctypes.byref(grid), K0.ctypes.data, ctypes.byref(op)))
    Ut = T(U)
    dk = torch.full((O.n_elem(nel),), np.nan, dtype=torch.float64, device="cuda")
    lib.check(L.pf_sensitivity_f64(op, lib.ptr(Ut), lib.ptr(dk), lib.stream()))
    assert rel(N(dk), O.process_dk(nel, K0, U)) < 1e-13
    L.pf_op_destroy(op)


@pytest.mark.parametrize("p", [1.0, 2.0, 3.0])
@pytest.mark.parametrize("heavyside", [False, True])
def test_penalize_whole_exponents_equal_pow(lib, p, heavyside):
    # the products against the general route, one ulp of the penalty away: r^(p eps) moves by at
    # most 3 * ln(1e9) * 2.2e-16 = 1.4e-14, pow and the products by a few ulp more
    from pyfantom_b200.Problem import penalize_device, simp_params
    rho = T(np.concatenate([[0.0, 1.0], np.random.default_rng(2).uniform(1e-9, 1, 5000)]))
    E, dE = penalize_device(rho, simp_params(p, 1e-9, 1.5, 3.0, 0.45, heavyside), True, True)
    E2, dE2 = penalize_device(rho, simp_params(np.nextafter(p, 9.0), 1e-9, 1.5, 3.0, 0.45, heavyside), True, True)
    assert np.allclose(N(E), N(E2), rtol=2e-14, atol=0)
    # (at rho = 0 with p = 1 the derivative is r^0 = 1 here and r^(2e-16) = 0 there)
    assert np.allclose(N(dE)[1:], N(dE2)[1:], rtol=2e-14, atol=0)
    # an empty projected density is exactly void in either route
    assert float(E[0]) == float(E2[0]) == 1e-9 * 1.5


@pytest.mark.parametrize("nel,n_level", [((8, 4, 4), 2), ((24, 12, 12), 2), ((16, 14, 14), 1), ((20, 20, 20), 1), ((40, 24), 2),
                                         ((120, 90), 1)])
def test_coarse_inverse(lib, nel, n_level):
    # one V-cycle against the oracle's (dense Cholesky of the coarsest operator), whose coarsest
    # orders run from two tiles through both routes (an order of 6,144 is the limit);
    # the two solves differ by the coarse operator's condition (up to 1e5) times 1e-16: 1e-9
    from conftest import unit_K0
    from pyfantom_b200 import workloads
    from pyfantom_b200.CUDA import MultiGrid, StructuredMesh2D, StructuredMesh3D, StructuredStiffnessKernel
    from pyfantom_b200.physics import LinearElasticity
    dim = len(nel)
    mesh = (StructuredMesh3D if dim == 3 else StructuredMesh2D)(*nel, *nel, physics=LinearElasticity(E=1.0, nu=0.3))
    kern = StructuredStiffnessKernel(mesh)
    wl = workloads.cantilever3d(*nel) if dim == 3 else workloads.mbb2d(*nel)
    kern.add_constraints(T(wl["fixed_dofs"], torch.int64))
    rng = np.random.default_rng(1)
    E = rng.uniform(0.1, 1.0, O.n_elem(nel))
    kern.set_rho(T(E))
    s = MultiGrid(mesh, kern, n_smooth=2, omega=0.6, n_level=n_level, coarse_op="stencil")
    s.setup()
    r = rng.standard_normal(kern.shape[0])
    r[wl["fixed_dofs"]] = 0.0
    z = N(s.vcycle(T(r), omega=0.4))
    assert rel(z, O.mg_vcycle(nel, unit_K0(dim), E, wl["fixed_dofs"], r, n_level=n_level, omega=0.4)) < 1e-9


@pytest.mark.parametrize("nel", [
    (2, 2, 2), (2, 3, 5), (7, 5, 82), (6, 4, 84), (5, 9, 169), (300, 62, 10), (301, 63, 85), (2, 600, 600), (31, 18)])
def test_restriction_rows(lib, nel):
    # 27 products and sums per value on each side, each within 1.1e-16 of the sum of magnitudes
    vf = np.random.default_rng(5).standard_normal(O.n_nodes(nel) * len(nel))
    grid, vft = lib.make_grid(nel), T(vf)
    out = torch.full((O.n_nodes(O.coarse_nel(nel)) * len(nel),), np.nan, dtype=torch.float64, device="cuda")
    lib.check(lib.load().pf_restrict_f64(ctypes.byref(grid), lib.ptr(vft), lib.ptr(out), lib.stream()))
    assert np.all(np.abs(N(out) - O.restrict(nel, vf)) <= 60 * 1.2e-16 * O.restrict(nel, np.abs(vf)))


@pytest.mark.parametrize("nel,nl,ns,kw", [
    ((8, 8, 8), 3, 2, {}), ((48, 24, 24), 3, 2, {}), ((24, 16, 8), 3, 1, {}), ((40, 24, 28), 3, 3, {}),
    ((36, 28, 32), 3, 2, {}), ((20, 18, 18), 2, 2, dict(coarse_op="stencil")), ((20, 20, 20), 2, 2, dict(coarse_op="stencil"))])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_vcycle_bottom(nel, nl, ns, kw, precision):
    # bottom levels of 27 to 1331 nodes: one launch where they fit shared memory, level by level beyond
    from test_solver_gpu import setup_problem
    from conftest import unit_K0
    from pyfantom_b200 import workloads
    wl = workloads.cantilever3d(*nel)
    mesh, kern, sol, fe = setup_problem(wl, nl, precision=precision, n_smooth=ns, **kw)
    kern.set_rho(T(wl["E"]))
    sol.setup()
    r = np.random.default_rng(0).standard_normal(kern.shape[0])
    r[wl["fixed_dofs"]] = 0.0
    z = N(sol.vcycle(T(r), omega=0.45))
    zr = O.mg_vcycle(nel, unit_K0(3), wl["E"], wl["fixed_dofs"], r, n_level=nl, n_smooth=ns, omega=0.45)
    # FP64: 2 ns products per level of conditioning below 1e5; FP32 carries 1e-7 per operation
    assert rel(z, zr) < (1e-10 if precision == "fp64" else 1e-4)


@pytest.mark.parametrize("nel,nl", [((16, 8, 8), 2), ((24, 12, 12), 2), ((48, 24, 24), 3), ((40, 24, 28), 3)])
@pytest.mark.parametrize("cut", [0.3, 0.6])
def test_vcycle_bottom_at_solid_and_void(nel, nl, cut):
    # solid 1 and void 1e-9 element by element, residuals of the size that each node's stiffness gives them.  The
    # coarsest operator is conditioned below 1e7 by its shift of 1e-6, the rest row by row: 1e-8
    from test_solver_gpu import setup_problem
    from conftest import unit_K0
    from pyfantom_b200 import workloads
    wl = workloads.cantilever3d(*nel)
    rng = np.random.default_rng(sum(nel))
    E = np.where(rng.uniform(size=O.n_elem(nel)) < cut, 1e-9, 1.0)
    mesh, kern, sol, fe = setup_problem(wl, nl)
    kern.set_rho(T(E))
    sol.setup()
    K0, fixed = unit_K0(3), wl["fixed_dofs"]
    u = rng.standard_normal(kern.shape[0])
    r = O.matvec(nel, K0, E, u, fixed)
    r[fixed] = 0.0
    z = N(sol.vcycle(T(r), omega=0.45))
    assert rel(z, O.mg_vcycle(nel, K0, E, fixed, r, n_level=nl, omega=0.45)) < 1e-8
