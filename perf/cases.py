"""Performance cases of the structured SIMP / MGCG library.

Each case is one call (or one short sequence of calls) that a topology-optimisation program
makes in its loop, through the library's public entry points: the Python object API of
``pyfantom_b200.CUDA`` and, for the steps that the object API only offers as part of a whole
optimiser iteration or of network training, the C ABI of ``include/pyfantom_b200.h``.

``op`` says which step a case is:

* ``matvec``   K(E) u on the stiffness kernel (``kernel.dot``): every solver's inner product.
* ``filter``   the density filter and its transpose, once each per SIMP iteration.
* ``gradient`` SIMP law, its derivative, the element sensitivity and the filter transpose:
               the gradient of the compliance once the displacements are known.
* ``oc``       one optimality-criteria update (``pf_oc_update_f64``).
* ``vcycle``   one multigrid V-cycle as a preconditioner application (``MultiGrid.vcycle``).
* ``solve``    a complete MGCG solve, hierarchy setup included, as in every SIMP iteration
               (the densities are new each time).
* ``direct``   the direct solve that small 2D problems use (``SPSOLVE``).
* ``conv``     one convolution layer of the learned form as a training step runs it: forward,
               input gradient and weight gradient on the tensor cores.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

PENALTY, VOID, NU = 3.0, 1e-9, 0.3
BETA, ETA = 2.0, 0.5  # Heaviside projection of the bridge workload
MOVE = 0.2
# Relative residual of the complete solves, as in the solver tests.  A displacement is only
# determined to about its solve's tolerance; at this one the forms agree to 1e-11.
TOL = 1e-10


# -----------------------------------------------------------------------------------------
# the cases
# -----------------------------------------------------------------------------------------
def listed():
    return [
        # the 2D MBB half-beam of the first configuration: the smallest product, all latency
        dict(name="matvec_mbb_120x40", op="matvec", nx=120, ny=40, nz=0, lx=120.0, ly=40.0, lz=0.0),
        # ragged counts and a box element that is no cube: a part meshed to its own dimensions
        dict(name="matvec_box_97x45x53", op="matvec", nx=97, ny=45, nz=53, lx=97.0, ly=54.0, lz=53.0),
        # the largest configuration (12.8 M DOF): the FP64 product of the outer CG
        dict(name="matvec_256x128x128", op="matvec", nx=256, ny=128, nz=128, lx=256.0, ly=128.0, lz=128.0),
        # filter pair of the 96x48x48 cantilever, rmin 2
        dict(name="filter_96x48x48_r2", op="filter", nx=96, ny=48, nz=48, rmin=2.0),
        # filter pair of the largest cantilever
        dict(name="filter_256x128x128_r2", op="filter", nx=256, ny=128, nz=128, rmin=2.0),
        # the differentiable bridge (rmin 2.5), with the projection switched on
        dict(name="gradient_bridge_128x64x64", op="gradient", nx=128, ny=64, nz=64, rmin=2.5, heavyside=True),
        # design update of the 192x96x96 cantilever
        dict(name="oc_192x96x96", op="oc", nx=192, ny=96, nz=96, volfrac=0.3),
        # preconditioner of the 192x96x96 precision form: FP32 V-cycle, BF16 element scales
        dict(name="vcycle_bf16_192x96x96", op="vcycle", nx=192, ny=96, nz=96, precision="mixed_bf16", n_level=5),
        # the plain FP64 drop-in at the size the reference quotes
        dict(name="solve_fp64_96x48x48", op="solve", nx=96, ny=48, nz=48, form="fp64", n_level=4),
        # the flagship: FP32 V-cycle and learned coarse space inside the FP64 CG
        dict(name="solve_learned_256x128x128", op="solve", nx=256, ny=128, nz=128, form="learned", n_level=5),
        # 2D MBB beam solved directly, as the reference's first example does
        dict(name="direct_mbb_60x20", op="direct", nx=60, ny=20),
        # last decoder layer of the network at its training grid and batch
        dict(name="conv_d1_64x32x32_b8", op="conv", batch=8, cin=48, cout=16, x=64, y=32, z=32, stride=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["matvec", "matvec", "filter", "gradient", "oc", "vcycle", "solve", "solve", "direct", "conv", "conv"])
    if op == "matvec" and rng.random() < 0.3:  # 2D
        nx, ny = _log(rng, 60, 1000), _log(rng, 20, 500)
        return dict(op=op, nx=nx, ny=ny, nz=0, lx=float(nx), ly=float(ny) * rng.choice([1.0, 1.25]), lz=0.0)
    # 3D parts about twice as long as wide
    w = _log(rng, 16, 126)
    nx, ny, nz = 2 * w + rng.randint(-7, 4), w + rng.randint(-3, 2), w + rng.randint(-3, 2)
    if op == "matvec":
        s = rng.choice([1.0, 1.0, 1.2])  # cube elements, or boxes longer along y
        return dict(op=op, nx=nx, ny=ny, nz=nz, lx=float(nx), ly=ny * s, lz=float(nz))
    if op == "filter":
        return dict(op=op, nx=nx, ny=ny, nz=nz, rmin=rng.choice([1.5, 2.0, 2.5]) if w < 80 else 2.0)
    if op == "gradient":
        return dict(op=op, nx=nx, ny=ny, nz=nz, rmin=rng.choice([1.5, 2.0, 2.5]) if w < 80 else 2.0,
                    heavyside=rng.random() < 0.5)
    if op == "oc":
        return dict(op=op, nx=nx, ny=ny, nz=nz, volfrac=rng.choice([0.2, 0.3, 0.5]))
    if op == "vcycle":
        return dict(op=op, nx=nx, ny=ny, nz=nz, precision=rng.choice(["fp64", "mixed", "mixed_bf16"]),
                    n_level=_levels(min(nx, ny, nz)))
    if op == "solve":  # counts that the hierarchy (and, in the learned form, the network) halves evenly
        form = rng.choice(["fp64", "mixed", "learned"])
        if form == "learned":
            p = _pool(w)
            lv, m = 3 + p // 2, max(2, w // (8 * p))
            return dict(op=op, nx=2 * m << lv, ny=m << lv, nz=m << lv, form=form, n_level=lv)
        lv = int(math.log2(w / 3.0))
        m = w >> lv
        return dict(op=op, nx=(2 * m + rng.choice([-1, 0, 1])) << lv, ny=m << lv, nz=m << lv, form=form, n_level=lv)
    if op == "direct":
        ny = rng.randint(8, 20)
        return dict(op=op, nx=ny * 3 - rng.randint(0, 4), ny=ny)
    cin, cout, stride = rng.choice([(8, 16, 1), (16, 16, 1), (16, 32, 2), (32, 32, 1), (32, 64, 2), (64, 48, 2),
                                    (160, 64, 1), (96, 32, 1), (48, 16, 1), (16, 3, 1)])
    top = 32 if cin * cout <= 1024 else 20
    x = _log(rng, 8, 2 * top)
    return dict(op="conv", batch=rng.randint(1, 8), cin=cin, cout=cout, x=x, y=_log(rng, 8, top), z=_log(rng, 8, top),
                stride=stride)


def _levels(n):
    """Halvings that leave at least three elements along the shortest axis."""
    lv = 1
    while n >> (lv + 1) >= 3:
        lv += 1
    return min(lv, 5)


def _pool(n):
    return 4 if n >= 96 else 2 if n >= 48 else 1


# -----------------------------------------------------------------------------------------
# inputs (made on the GPU from the seed alone)
# -----------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) + 1)


def _smoothed(nel, seed, sigma=2.0):
    """uniform(0.001, 1) in element order, Gaussian-smoothed with sigma 2 (edges replicated):
    the density field of the cantilever and bridge configurations."""
    x = torch.rand(nel, generator=_gen(seed), device="cuda", dtype=torch.float64) * 0.999 + 0.001
    r = int(4 * sigma)
    t = torch.arange(-r, r + 1, device="cuda", dtype=torch.float64)
    w = torch.exp(-0.5 * (t / sigma) ** 2)
    w = (w / w.sum()).tolist()
    for a in range(len(nel)):
        idx = torch.arange(nel[a], device="cuda")
        y = torch.zeros_like(x)
        for q in range(2 * r + 1):
            y += w[q] * x.index_select(a, (idx + q - r).clamp(0, nel[a] - 1))
        x = y
    return x.reshape(-1)


def _nel(c):
    return (c["nx"], c["ny"], c["nz"]) if c.get("nz") else (c["nx"], c["ny"])


def _cantilever(nel, seed):
    """(constrained DOFs, load): clamped face x = 0, unit load over the lower edge of the far
    face, its direction from the seed."""
    nx, ny, nz = (v + 1 for v in nel)
    j, k = torch.meshgrid(torch.arange(ny, device="cuda"), torch.arange(nz, device="cuda"), indexing="ij")
    fixed = (k + nz * nx * j).reshape(-1)
    cons = (fixed[:, None] * 3 + torch.arange(3, device="cuda")).reshape(-1)
    d = torch.randn(3, generator=_gen(seed + 7), device="cuda", dtype=torch.float64)
    d = d * 0.3
    d[1] = -1.0
    rhs = torch.zeros(nx * ny * nz, 3, device="cuda", dtype=torch.float64)
    edge = torch.arange(nz, device="cuda") + nz * (nx - 1)
    rhs[edge] = d / nz
    return cons, rhs.reshape(-1)


def _mbb(nel):
    """Roller on the left edge and at the lower right corner, unit load at the upper left."""
    nx, ny = nel[0] + 1, nel[1] + 1
    left = torch.arange(ny, device="cuda") * nx
    cons = torch.cat([left * 2, torch.tensor([(nx - 1) * 2 + 1], device="cuda")])
    rhs = torch.zeros(nx * ny * 2, device="cuda", dtype=torch.float64)
    rhs[(ny - 1) * nx * 2 + 1] = -1.0
    return cons, rhs


def _mesh(c):
    from pyfantom_b200.CUDA import StructuredMesh2D, StructuredMesh3D
    from pyfantom_b200.physics import LinearElasticity
    nel = _nel(c)
    dims = [c.get(k) or float(n) for k, n in zip(("lx", "ly", "lz"), nel)]
    return (StructuredMesh3D if len(nel) == 3 else StructuredMesh2D)(*nel, *dims,
                                                                     physics=LinearElasticity(E=1.0, nu=NU))


def _kernel(mesh, cons):
    from pyfantom_b200.CUDA import StructuredStiffnessKernel
    kern = StructuredStiffnessKernel(mesh)
    kern.set_constraints(cons)
    return kern


def _displacement(nel, seed):
    """A bending-like field with noise: what the product and the sensitivity see in a solve."""
    dim = len(nel)
    n = int(np.prod([v + 1 for v in nel]))
    u = torch.randn(n, dim, generator=_gen(seed + 3), device="cuda", dtype=torch.float64)
    i = (torch.arange(n, device="cuda") // (nel[2] + 1 if dim == 3 else 1)) % (nel[0] + 1)
    bend = (i.double() / nel[0]) ** 2
    u = 0.05 * u
    u[:, 1] -= bend
    u[:, 0] += 0.3 * bend
    return u.reshape(-1)


def _conv_inputs(c, seed):
    g = _gen(seed)
    n, ci, co, s = c["batch"], c["cin"], c["cout"], c["stride"]
    xs = (c["x"], c["y"], c["z"])
    os_ = tuple((v - 1) // s + 1 for v in xs)

    def rnd(*shape):
        return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32)

    x = torch.relu(rnd(n, ci, *xs))  # the layer before ends in a ReLU
    w = rnd(co, ci, 3, 3, 3) * math.sqrt(2.0 / (27 * ci))
    b = 0.1 * rnd(co)
    dy = rnd(n, co, *os_) / math.sqrt(n * np.prod(os_))
    return x, w, b, dy


def _oc_inputs(c, seed):
    nel = _nel(c)
    x = _smoothed(nel, seed)
    x = (x * (c["volfrac"] / x.mean())).clamp(0.0, 1.0)
    # a compliance gradient: negative, over several decades
    s = _smoothed(nel, seed + 5)
    df = -torch.exp(24.0 * (s - s.mean())) * (0.05 + x * x)
    dg = torch.full_like(x, 1.0 / x.numel())
    return x, df, dg


def prepare(case, seed):
    from pyfantom_b200 import _lib
    c, op, st = case, case["op"], {"op": case["op"], "case": case}
    if op == "matvec":
        nel = _nel(c)
        mesh = _mesh(c)
        cons = _mbb(nel)[0] if len(nel) == 2 else _cantilever(nel, seed)[0]
        kern = _kernel(mesh, cons)
        kern.set_rho(_smoothed(nel, seed).pow(PENALTY).clamp(VOID, 1.0))
        st.update(kern=kern, u=_displacement(nel, seed))
    elif op in ("filter", "gradient"):
        from pyfantom_b200.CUDA import FiniteElement, MinimumCompliance, MultiGrid, StructuredFilter3D
        nel = _nel(c)
        mesh = _mesh(c)
        st["filter"] = StructuredFilter3D(mesh, c["rmin"])
        x = _smoothed(nel, seed)
        if op == "filter":
            st.update(x=x, v=-_smoothed(nel, seed + 5))
        else:
            kern = _kernel(mesh, _cantilever(nel, seed)[0])
            fe = FiniteElement(mesh, kern, MultiGrid(mesh, kern, n_level=1))
            st["problem"] = MinimumCompliance(fe, st["filter"], E_mul=[1.0], void=VOID, penalty=PENALTY,
                                              volume_fraction=[0.2], heavyside=c["heavyside"], beta=BETA, eta=ETA)
            st.update(x=x, U=_displacement(nel, seed), kern=kern)
    elif op == "oc":
        x, df, dg = _oc_inputs(c, seed)
        lib = _lib.load()
        work = torch.empty(int(lib.pf_oc_workspace_size(x.numel())), device="cuda", dtype=torch.float64)
        st.update(lib=lib, x=x, df=df, dg=dg, work=work, out=torch.empty_like(x), info=(ctypes.c_double * 3)())
    elif op in ("vcycle", "solve"):
        from pyfantom_b200.CUDA import MultiGrid
        nel = _nel(c)
        mesh = _mesh(c)
        cons, rhs = _cantilever(nel, seed)
        kern = _kernel(mesh, cons)
        E = _smoothed(nel, seed).pow(PENALTY).clamp(VOID, 1.0)
        kw = dict(maxiter=1000, n_smooth=2, omega=0.6, n_level=c["n_level"])
        if op == "vcycle":
            solver = MultiGrid(mesh, kern, precision=c["precision"], **kw)
            kern.set_rho(E)
            solver.setup()
            r = torch.randn(rhs.shape, generator=_gen(seed + 9), device="cuda", dtype=torch.float64)
            r[cons] = 0.0
            st.update(solver=solver, r=r, single=c["precision"] != "fp64")
        else:
            form = c["form"]
            kw["tol"] = TOL
            if form == "learned":
                from pyfantom_b200.learned import LearnedCoarseSpace, WarmStartNet
                kw.update(coarse_correction=LearnedCoarseSpace(WarmStartNet.load(), pool=_pool(min(nel))))
            if form != "fp64":
                kw.update(precision="mixed", fixed_omega=0.5)
            st.update(solver=MultiGrid(mesh, kern, **kw), rhs=rhs, E=E)
    elif op == "direct":
        from pyfantom_b200.CUDA import SPSOLVE
        nel = _nel(c)
        cons, rhs = _mbb(nel)
        kern = _kernel(_mesh(c), cons)
        st.update(solver=SPSOLVE(kern), rhs=rhs, E=_smoothed(nel, seed).pow(PENALTY).clamp(VOID, 1.0))
    else:
        x, w, b, dy = _conv_inputs(c, seed)
        lib = _lib.load()
        n, ci, co, s = c["batch"], c["cin"], c["cout"], c["stride"]
        nw = lib.pf_cnn_conv3d_bwd_weight_tc_workspace(n, ci, c["x"], c["y"], c["z"], co, s)
        st.update(lib=lib, x=x, w=w, b=b, dy=dy, y=torch.empty_like(dy), dx=torch.empty_like(x),
                  dw=torch.empty_like(w), db=torch.empty_like(b),
                  work=torch.empty(int(nw), device="cuda", dtype=torch.float32),
                  err=torch.zeros(1, device="cuda", dtype=torch.int32))
    return st


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


# -----------------------------------------------------------------------------------------
# one pass
# -----------------------------------------------------------------------------------------
def run(st):
    op = st["op"]
    if op == "matvec":
        return st["kern"].dot(st["u"])
    if op == "filter":
        return st["filter"].dot(st["x"]), st["filter"].T @ st["v"]
    if op == "gradient":
        p = st["problem"]
        rho = st["filter"].dot(st["x"])
        E, dE = p.penalize(rho), p.penalize_grad(rho)
        return E, st["filter"].T @ (dE * st["kern"].process_grad(st["U"]))
    if op == "oc":
        x, out = st["x"], st["out"]
        status = st["lib"].pf_oc_update_f64(x.numel(), _ptr(x), _ptr(st["df"]), _ptr(st["dg"]), st["case"]["volfrac"],
                                            MOVE, _ptr(out), _ptr(st["work"]), st["info"], _stream())
        if status:
            raise RuntimeError("pf_oc_update_f64: %d" % status)
        return out
    if op == "vcycle":  # the FP32 V-cycle's result holds single-precision values
        z = st["solver"].vcycle(st["r"])
        return z.float() if st["single"] else z
    if op == "solve":
        return st["solver"].solve(st["rhs"], rho=st["E"], use_last=False)[0]
    if op == "direct":
        return st["solver"].solve(st["rhs"], rho=st["E"])[0]
    c, lib, s = st["case"], st["lib"], _stream()
    dims = (c["batch"], c["cin"], c["x"], c["y"], c["z"])
    status = lib.pf_cnn_conv3d_fwd_tc(_ptr(st["x"]), *dims, _ptr(st["w"]), _ptr(st["b"]), c["cout"], c["stride"], 1,
                                      _ptr(st["y"]), _ptr(st["err"]), s)
    status |= lib.pf_cnn_conv3d_bwd_data_tc(_ptr(st["dy"]), *dims, _ptr(st["w"]), c["cout"], c["stride"], 0,
                                            _ptr(st["dx"]), _ptr(st["err"]), s)
    status |= lib.pf_cnn_conv3d_bwd_weight_tc(_ptr(st["x"]), _ptr(st["dy"]), *dims, c["cout"], c["stride"],
                                              _ptr(st["dw"]), _ptr(st["db"]), _ptr(st["work"]), _ptr(st["err"]), s)
    if status:
        raise RuntimeError("convolution: %d" % status)
    return st["y"], st["dx"], st["dw"], st["db"]


# -----------------------------------------------------------------------------------------
# what a pass cannot do without
# -----------------------------------------------------------------------------------------
def _taps(rmin):
    n = int(math.ceil(rmin))
    return [(a, b, d, rmin - math.sqrt(a * a + b * b + d * d)) for a in range(-n, n + 1) for b in range(-n, n + 1)
            for d in range(-n, n + 1) if a * a + b * b + d * d < rmin * rmin]


def work(case):
    c, op = case, case["op"]
    if op == "conv":
        s = c["stride"]
        vi = c["x"] * c["y"] * c["z"]
        vo = math.prod((c[k] - 1) // s + 1 for k in "xyz")
        wn = 27 * c["cin"] * c["cout"]
        byte = 4 * (c["batch"] * (2 * c["cin"] * vi + 2 * c["cout"] * vo) + 2 * wn)
        return {"bytes": byte, "flops": 6 * c["batch"] * vo * wn}
    nel = _nel(c)
    dim = len(nel)
    ne = math.prod(nel)
    D = dim * math.prod(v + 1 for v in nel)
    if op == "matvec":  # u, E in, y out; the Walsh form of the element product
        return {"bytes": 16 * D + 8 * ne, "flops": (150 if dim == 3 else 128) * ne}
    if op == "filter":
        return {"bytes": 32 * ne, "flops": 4 * len(_taps(c["rmin"])) * ne}
    if op == "gradient":  # x, U in; E and the gradient out
        return {"bytes": 8 * D + 24 * ne, "flops": (4 * len(_taps(c["rmin"])) + 200) * ne}
    if op == "oc":  # x, df, dg in, x_new out
        return {"bytes": 32 * ne, "flops": 90 * 6 * ne}
    if op == "direct":  # banded Cholesky of the free DOFs
        band = 2 * (min(nel) + 2)
        return {"bytes": 8 * (2 * D + ne), "flops": D * band * band}
    # one V-cycle: four fine products with their operands, a seventh of that below
    t = 4 if c.get("precision", "mixed") != "fp64" and c.get("form") != "fp64" else 8
    cyc = 8.0 / 7.0 * (4 * (2 * t * D + t * ne) + 8 * t * D)
    flops = 8.0 / 7.0 * 4 * 160 * ne
    if op == "vcycle":
        return {"bytes": cyc + 16 * D, "flops": flops}
    its = 60  # iterations, of order: the V-cycle, the FP64 product, two axpys and the dots
    return {"bytes": its * (cyc + 16 * D + 8 * ne + 56 * D), "flops": its * (flops + 150 * ne)}


# -----------------------------------------------------------------------------------------
# the same results in 64 bits, by plain torch
# -----------------------------------------------------------------------------------------
_CORNERS = ((0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1))


def _element_matrix(h):
    """Stiffness of an isotropic box (plane stress in 2D), two Gauss points per axis."""
    dim = len(h)
    corners = np.array([q[:dim] for q in _CORNERS[:2 ** dim]], dtype=float)
    mu = 0.5 / (1 + NU)
    lam = NU / ((1 + NU) * (1 - 2 * NU)) if dim == 3 else NU / (1 - NU * NU)
    g = [0.5 - 0.5 / math.sqrt(3.0), 0.5 + 0.5 / math.sqrt(3.0)]
    K = np.zeros((2 ** dim, dim, 2 ** dim, dim))
    for p in np.array(np.meshgrid(*[g] * dim)).reshape(dim, -1).T:
        f = np.where(corners == 1, p, 1 - p)  # one-dimensional shape functions
        dN = np.stack([np.where(corners[:, a] == 1, 1.0, -1.0) / h[a] * np.prod(np.delete(f, a, 1), axis=1)
                       for a in range(dim)], axis=1)
        wt = math.prod(h) / 2 ** dim
        K += wt * (lam * np.einsum("ai,bj->aibj", dN, dN) + mu * np.einsum("aj,bi->aibj", dN, dN))
        for i in range(dim):
            K[:, i, :, i] += wt * mu * dN @ dN.T
    return torch.as_tensor(K.reshape(dim * 2 ** dim, -1), device="cuda")


def _connectivity(nel):
    dim = len(nel)
    ax = torch.meshgrid(*[torch.arange(n, device="cuda") for n in nel], indexing="ij")
    nn = [v + 1 for v in nel]
    nodes = []
    for q in _CORNERS[:2 ** dim]:
        p = [a + o for a, o in zip(ax, q)]
        nodes.append((p[2] + nn[2] * (p[0] + nn[0] * p[1]) if dim == 3 else p[0] + nn[0] * p[1]).reshape(-1))
    return torch.stack(nodes, 1)


def _exact_matvec(nel, h, E, u, cons):
    dim = len(nel)
    K = _element_matrix(h)
    conn = _connectivity(nel)
    free = u.clone()
    free[cons] = 0.0
    y = torch.zeros_like(u).reshape(-1, dim)
    for part in torch.arange(conn.shape[0], device="cuda").split(1 << 20):
        ue = free.reshape(-1, dim)[conn[part]].reshape(len(part), -1)
        ye = (ue @ K) * E[part, None]
        y.index_add_(0, conn[part].reshape(-1), ye.reshape(-1, dim))
    y = y.reshape(-1)
    y[cons] = u[cons]
    return y


def _exact_filter(nel, rmin, x, transpose):
    """x, or its transpose applied: taps of the cone, normalised by the sum inside the mesh."""
    def taps(v):
        n = int(math.ceil(rmin))
        p = torch.nn.functional.pad(v.reshape(1, 1, *nel), (n,) * 6)[0, 0]
        out = torch.zeros(nel, device="cuda", dtype=torch.float64)
        for a, b, d, wt in _taps(rmin):
            out += wt * p[n + a:n + a + nel[0], n + b:n + b + nel[1], n + d:n + d + nel[2]]
        return out.reshape(-1)
    norm = taps(torch.ones_like(x))
    return taps(x / norm) if transpose else taps(x) / norm


def exact(case, seed):
    c, op = case, case["op"]
    if op == "matvec":
        nel = _nel(c)
        h = [c[k] / n for k, n in zip(("lx", "ly", "lz"), nel)]
        cons = _mbb(nel)[0] if len(nel) == 2 else _cantilever(nel, seed)[0]
        E = _smoothed(nel, seed).pow(PENALTY).clamp(VOID, 1.0)
        return _exact_matvec(nel, h, E, _displacement(nel, seed), cons)
    if op == "filter":
        nel = _nel(c)
        return (_exact_filter(nel, c["rmin"], _smoothed(nel, seed), False),
                _exact_filter(nel, c["rmin"], -_smoothed(nel, seed + 5), True))
    if op == "gradient":
        nel = _nel(c)
        rho = _exact_filter(nel, c["rmin"], _smoothed(nel, seed), False)
        H, dH = rho, 1.0
        if c["heavyside"]:
            den = math.tanh(BETA * ETA) + math.tanh(BETA * (1 - ETA))
            t = torch.tanh(BETA * (rho - ETA))
            H, dH = (math.tanh(BETA * ETA) + t) / den, BETA * (1 - t * t) / den
        E = H.pow(PENALTY).clamp(VOID, 1.0)
        dE = PENALTY * H.pow(PENALTY - 1) * dH
        conn, K = _connectivity(nel), _element_matrix([1.0, 1.0, 1.0])
        U = _displacement(nel, seed).reshape(-1, 3)
        dk = torch.cat([-((U[q].reshape(len(q), -1) @ K) * U[q].reshape(len(q), -1)).sum(1) for q in conn.split(1 << 20)])
        return E, _exact_filter(nel, c["rmin"], dE * dk, True)
    if op == "oc":
        x, df, dg = _oc_inputs(c, seed)
        oc = x * torch.sqrt((-df / dg).clamp(min=0.0))
        lo, hi = (x - MOVE).clamp(0.0, 1.0), (x + MOVE).clamp(0.0, 1.0)
        l1, l2, new = 1e-9, 1e9, x
        while (l2 - l1) / (l2 + l1) > 1e-8:
            mid = 0.5 * (l1 + l2)
            new = torch.maximum(lo, torch.minimum(hi, oc / mid))
            if float(torch.dot(dg, new)) <= c["volfrac"]:
                l2 = mid
            else:
                l1 = mid
        return new
    if op == "direct":
        nel = _nel(c)
        cons, rhs = _mbb(nel)
        E = _smoothed(nel, seed).pow(PENALTY).clamp(VOID, 1.0)
        D = rhs.numel()
        conn, K = _connectivity(nel), _element_matrix([1.0, 1.0])
        dofs = (conn[:, :, None] * 2 + torch.arange(2, device="cuda")).reshape(len(conn), 8)
        A = torch.zeros(D * D, device="cuda", dtype=torch.float64)
        A.index_add_(0, (dofs[:, :, None] * D + dofs[:, None, :]).reshape(-1), (E[:, None, None] * K).reshape(-1))
        A = A.reshape(D, D)
        free = torch.ones(D, device="cuda", dtype=torch.bool)
        free[cons] = False
        f = free.nonzero().reshape(-1)
        out = rhs.clone()
        out[f] = torch.linalg.solve(A[f][:, f], rhs[f])
        return out
    if op == "conv":
        x, w, b, dy = (t.double().requires_grad_(k < 3) for k, t in enumerate(_conv_inputs(c, seed)))
        y = torch.nn.functional.conv3d(x, w, b, stride=c["stride"], padding=1)
        dx, dw, db = torch.autograd.grad(y, (x, w, b), dy)
        return torch.relu(y), dx, dw, db
    return None  # V-cycles and complete solves: no closed form
