"""The work that a user of this framework has it do, as measurable cases.

Every case is one call (or one solve) through the package's public entry points, on the
meshes, discretisations and sizes of the repository's own workloads:

  assemble   NavierStokesFV1.assemble_defect / assemble_jacobian / assemble_defect_jacobian
  spmv       NavierStokesFV1.bsr_mv
  linear     NavierStokesFV1.linear_solve with a bounded number of iterations
  newton     NavierStokesFV1.newton_solve with a bounded number of steps
  batch      CavityBatch.solve (the batched Newton)
  predict    CoordinateMLP.predict (the learned warm start)
  grad       CoordinateMLP.loss_grad (its training step)

``listed()`` gives the named cases, ``draw(rng)`` one more of the same ranges, ``prepare``
what a program holds before the call, ``run`` one pass, ``work`` the bytes and operations
that one pass cannot do without, ``exact`` the result in plain 64-bit torch.
"""
import functools
import math

import numpy as np
import torch

from plugin_navierstokes_gb300 import NavierStokesFV1, mesh
from plugin_navierstokes_gb300.warm_start import CavityBatch, CoordinateMLP

TRI, QUAD, HEX = 2, 3, 8
NSH = {TRI: 3, QUAD: 4, HEX: 8}
MLP_WIDTH, MLP_FEATURES, MLP_PARAMS = 256, 64, 220931


# ---- the cases -----------------------------------------------------------------


def listed():
    return [
        # the flagship assembly: one Newton step's FP64 defect and Jacobian on the 64^3 cavity
        dict(name="hex64_defect_jacobian_f64", kind="assemble", what="both", mesh="hex", n=64, prec="f64", upwind="lps", stab="flow", transient=False, walls=False),
        # the same step in the FP32-Jacobian mode on a distorted mesh of odd size, inside an implicit Euler step
        dict(name="hexj41_defect_jacobian_f32", kind="assemble", what="both", mesh="hexj", n=41, prec="f32", upwind="full", stab="flow", transient=True, walls=False),
        # the defect of a line search in the transient triangle workload (2 x 1024^2 triangles)
        dict(name="tri1024_defect_f64", kind="assemble", what="defect", mesh="tri", n=1024, prec="f64", upwind="full", stab="fields", transient=True, walls=True),
        # the Jacobian of that workload as its Newton loop stores it
        dict(name="tri1024_jacobian_f32", kind="assemble", what="jacobian", mesh="tri", n=1024, prec="f32", upwind="full", stab="fields", transient=True, walls=False),
        # the smallest call: one 32^2 cavity, where launches count
        dict(name="quad32_defect_jacobian_f64", kind="assemble", what="both", mesh="quad", n=32, prec="f64", upwind="full", stab="flow", transient=False, walls=True),
        # the product with an FP64 3D matrix (a user's own Krylov method, GMRES)
        dict(name="hex48_spmv_f64", kind="spmv", mesh="hex", n=48, prec="f64"),
        # the inner solver of the transient workload: BiCGStab, FP32 matrix, FP64 vectors
        dict(name="tri700_bicgstab_f32", kind="linear", mesh="tri", n=700, prec="f32", upwind="full", stab="fields", transient=True, solver="bicgstab", iters=10),
        # the other linear solver, FP64, on a cavity of the batched workload's size
        dict(name="quad192_gmres_f64", kind="linear", mesh="quad", n=192, prec="f64", upwind="full", stab="flow", transient=False, solver="gmres", iters=45),
        # a whole Newton call on one 64^2 cavity from rest (two steps, each with a bounded solve)
        dict(name="quad64_newton_f64", kind="newton", mesh="quad", n=64, prec="f64", upwind="full", stab="flow", transient=False, solver="gmres", iters=30, steps=2),
        # a batch of uneven cavities solved together in the FP32-Jacobian mode
        dict(name="batch12_cavities_f32", kind="batch", instances=12, sizes="32,48,64", prec="f32"),
        # the network's initial iterate of 32 cavities of 128^2 cells
        dict(name="predict32_cavity128", kind="predict", instances=32, n=128),
        # one training step's loss and gradient: 64 instances x 1024 nodes
        dict(name="grad64x1024", kind="grad", slots=64, points=1024),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["assemble", "assemble", "assemble", "assemble", "spmv", "linear", "linear", "newton", "batch", "predict", "grad"])
    if kind in ("assemble", "spmv", "linear", "newton"):
        m = rng.choice(["hex", "hexj", "tri", "quad"] if kind != "newton" else ["quad", "tri"])
        hi = {"assemble": {"hex": 60, "hexj": 44, "tri": 900, "quad": 900}, "spmv": {"hex": 48, "hexj": 48, "tri": 900, "quad": 900},
              "linear": {"hex": 30, "hexj": 30, "tri": 600, "quad": 400}, "newton": {"quad": 90, "tri": 60}}[kind][m]
        c = dict(kind=kind, mesh=m, n=_log(rng, 5 if m in ("hex", "hexj") else 17, hi), prec=rng.choice(["f64", "f32"]))
        if kind == "spmv":
            return c
        # the ray test of LPS has a closed form on affine elements only: exact() has it there
        c["upwind"] = rng.choice(["full", "no"] if m == "hexj" else ["full", "lps"])
        c["stab"] = rng.choice(["flow", "fields"])
        c["transient"] = rng.random() < 0.5
        if kind == "assemble":
            c["what"] = rng.choice(["both", "both", "defect", "jacobian"])
            c["walls"] = rng.random() < 0.5
            return c
        if kind == "newton":
            c.update(solver="gmres", iters=rng.randrange(12, 31), steps=2, prec="f64")
            return c
        c["solver"] = rng.choice(["bicgstab", "gmres"])
        c["iters"] = rng.randrange(6, 11) if c["solver"] == "bicgstab" else rng.randrange(10, 61)
        return c
    if kind == "batch":
        return dict(kind="batch", instances=rng.randrange(3, 13), sizes=rng.choice(["32,48", "32,64", "48,64", "32,48,64"]), prec="f32")
    if kind == "predict":
        return dict(kind="predict", instances=_log(rng, 1, 32), n=_log(rng, 8, 128))
    return dict(kind="grad", slots=_log(rng, 2, 64), points=_log(rng, 33, 1024))


# ---- meshes and states ---------------------------------------------------------


@functools.lru_cache(maxsize=4)
def _mesh(kind, n):
    """(element type, coordinates, connectivity) of an n-cell mesh of the unit square or cube."""
    if kind == "tri":
        return mesh.jittered_triangles(n, seed=2)
    if kind == "quad":
        return mesh.structured_quads(n)
    t, x, c = mesh.structured_hexes(n)
    if kind == "hexj":
        # inner nodes moved by up to 0.15 cells: no element is a parallelepiped
        inner = np.all((x > 1e-9) & (x < 1 - 1e-9), axis=1)
        x = x + (np.random.RandomState(2).rand(*x.shape) * 2 - 1) * (0.15 / n) * inner[:, None]
    return t, x, c


@functools.lru_cache(maxsize=4)
def _walls(kind, n):
    return mesh.cavity_dirichlet(_mesh(kind, n)[1])


def _state(x, seed, moved=0.0):
    """A smooth velocity and pressure on the nodes x (device), a few seeded modes."""
    dim = x.shape[1]
    r = np.random.RandomState(seed)
    u = torch.zeros(x.shape[0], dim + 1, dtype=torch.float64, device=x.device)
    for f in range(dim + 1):
        for _ in range(6):
            k = r.randint(1, 6, size=dim) * math.pi
            a, ph = r.uniform(-0.5, 0.5), r.uniform(0, 2 * math.pi, size=dim)
            w = torch.full((x.shape[0],), a, dtype=torch.float64, device=x.device)
            for d in range(dim):
                w = w * torch.sin(x[:, d] * k[d] + ph[d] + moved)
            u[:, f] += w
    return u.reshape(-1).contiguous()


def _iterate(case, x, seed, moved=0.0):
    """The state of a Newton iterate: with walls it has their values."""
    u = _state(x, seed, moved)
    if case.get("walls", True):
        rows, vals = _walls(case["mesh"], case["n"])
        u[torch.from_numpy(rows.astype(np.int64)).to(x.device)] = torch.from_numpy(vals).to(x.device)
    return u


def _nu(case):
    return 0.001 if case["transient"] else (0.0025 if case["mesh"].startswith("hex") else 0.01)


def _dt(case):
    return 0.01 if case["transient"] else 0.0


def _disc(case):
    t, x, c = _mesh(case["mesh"], case["n"])
    d = NavierStokesFV1("u,v,w,p" if x.shape[1] == 3 else "u,v,p", "Inner")
    if "upwind" in case:
        d.set_kinematic_viscosity(_nu(case))
        d.set_upwind(case["upwind"])
        d.set_stabilization(case["stab"])
    d.set_mesh(t, x, c)
    if case.get("walls", "upwind" in case):
        d.set_dirichlet(*_walls(case["mesh"], case["n"]))
    return d


def _dtype(case):
    return torch.float64 if case["prec"] == "f64" else torch.float32


# ---- one pass ------------------------------------------------------------------


def prepare(case, seed):
    k = case["kind"]
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    s = dict(case=case)
    if k in ("assemble", "spmv", "linear", "newton"):
        d = s["disc"] = _disc(case)
        nnz = d.pattern_info()["nnz_blocks"]
        b = d.dim + 1
        nv = d.n_nodes * b
    if k == "assemble" or (k in ("linear", "newton")):
        x = torch.from_numpy(_mesh(case["mesh"], case["n"])[1]).cuda()
        s["u"] = _iterate(case, x, seed)
        s["u_old"] = _iterate(case, x, seed, 0.02) if case["transient"] else None
    if k == "assemble":
        s["d"] = torch.empty(nv, dtype=torch.float64, device="cuda")
        if case["what"] != "defect":
            s["vals"] = torch.empty(nnz * b * b, dtype=_dtype(case), device="cuda")
    elif k == "spmv":
        s["vals"] = torch.randn(nnz * b * b, generator=g, dtype=_dtype(case), device="cuda")
        s["x"] = torch.randn(nv, generator=g, dtype=torch.float64, device="cuda")
        s["y"] = torch.empty_like(s["x"])
    elif k == "linear":
        s["vals"] = torch.empty(nnz * b * b, dtype=_dtype(case), device="cuda")
        d.assemble_jacobian(s["u"], s["vals"], s["u_old"], _dt(case))
        rhs = torch.randn(nv, generator=g, dtype=torch.float64, device="cuda")
        s["rhs"] = rhs / rhs.norm()
        s["x"] = torch.empty_like(rhs)
    elif k == "newton":
        # from a state near rest, as the first step of a continuation
        s["start"] = 0.05 * s["u"]
        s["u_old"] = None if s["u_old"] is None else s["start"].clone()
    elif k == "batch":
        r = np.random.RandomState(seed)
        sizes = [int(v) for v in case["sizes"].split(",")]
        n = np.array([sizes[i % len(sizes)] for i in range(case["instances"])])
        re = np.exp(r.uniform(math.log(10.0), math.log(400.0), size=n.size))
        s["batch"] = CavityBatch(n, re, r.uniform(0.5, 2.0, size=n.size))
        s["u"] = s["batch"].zeros()
    elif k == "predict":
        r = np.random.RandomState(seed)
        n, nn = case["instances"], (case["n"] + 1) ** 2
        s["net"] = CoordinateMLP(max_points=262144, max_slots=256, seed=seed)
        s["net"].set_params(_params(seed))
        xy = torch.from_numpy(mesh.structured_quads(case["n"])[1].astype(np.float32)).cuda()
        s["xy"] = xy.repeat(n, 1).contiguous()
        s["ptr"] = np.arange(n + 1, dtype=np.int32) * nn
        s["cond"] = r.uniform(-1, 1, size=(n, 2)).astype(np.float32)
        s["lid"] = r.uniform(0.5, 2.0, size=n).astype(np.float32)
        s["u"] = torch.empty(n * nn * 3, dtype=torch.float64, device="cuda")
    elif k == "grad":
        n = case["slots"] * case["points"]
        s["net"] = CoordinateMLP(max_points=65536, max_slots=256, seed=seed)
        s["net"].set_params(_params(seed))
        s["xy"] = torch.rand(n, 2, generator=g, dtype=torch.float32, device="cuda")
        s["target"] = torch.randn(n, 3, generator=g, dtype=torch.float32, device="cuda") * 0.3
        s["ptr"] = np.arange(case["slots"] + 1, dtype=np.int32) * case["points"]
        s["cond"] = np.random.RandomState(seed).uniform(-1, 1, size=(case["slots"], 2)).astype(np.float32)
        s["grad"] = torch.empty(s["net"].num_params, dtype=torch.float32, device="cuda")
    return s


def run(s):
    c = s["case"]
    k = c["kind"]
    if k == "assemble":
        u, uo, dt = s["u"], s["u_old"], _dt(c)
        if c["what"] == "both":
            s["disc"].assemble_defect_jacobian(u, s["d"], s["vals"], uo, dt)
            return [s["d"], s["vals"]]
        if c["what"] == "defect":
            s["disc"].assemble_defect(u, s["d"], uo, dt)
            return [s["d"]]
        s["disc"].assemble_jacobian(u, s["vals"], uo, dt)
        return [s["vals"]]
    if k == "spmv":
        s["disc"].bsr_mv(s["vals"], s["x"], s["y"])
        return [s["y"]]
    if k == "linear":
        s["disc"].linear_solve(s["vals"], s["rhs"], s["x"], lin_rtol=1e-12, lin_max_iter=c["iters"], linear_solver=c["solver"], gmres_restart=30,
                               raise_on_error=False)
        return [s["x"]]
    if k == "newton":
        u = s["u"].copy_(s["start"])
        s["disc"].newton_solve(u, s["u_old"], dt=_dt(c), rtol=1e-12, max_iter=c["steps"], lin_rtol=1e-12, lin_max_iter=c["iters"], jacobian_prec=c["prec"],
                               linear_solver=c["solver"], raise_on_error=False)
        return [u]
    if k == "batch":
        u = s["u"].zero_()
        s["batch"].solve(u, jacobian_prec=c["prec"], rtol=1e-12)
        return [u]
    if k == "predict":
        s["net"].predict(s["xy"], s["ptr"], s["cond"], s["lid"], s["u"])
        return [s["u"]]
    loss = s["net"].loss_grad(s["xy"], s["ptr"], s["cond"], s["target"], s["grad"])
    return [loss, s["grad"]]


# ---- what a pass cannot do without -----------------------------------------------


@functools.lru_cache(maxsize=None)
def _counts(kind, n):
    """(nodes, elements, matrix blocks, corners, dim) of a mesh without building it (tri: its mean of 7 blocks a row)."""
    m = n + 1
    if kind == "tri":
        return m * m, 2 * n * n, m * m + 2 * (3 * n * n + 2 * n), 3, 2
    if kind == "quad":
        return m * m, n * n, (3 * n + 1) ** 2, 4, 2
    return m**3, n**3, (3 * n + 1) ** 3, 8, 3


def work(case):
    k = case["kind"]
    if k in ("assemble", "spmv", "linear", "newton"):
        nodes, elems, nnz, nsh, dim = _counts(case["mesh"], case["n"])
        b, vb = dim + 1, 8 if case["prec"] == "f64" else 4
        vec, mat = nodes * b * 8.0, nnz * b * b * float(vb)
        elem_in = elems * nsh * 4.0 + nodes * dim * 8.0 + vec * (2 if case.get("transient") else 1)
        # per SCVF: its state (about 60 operations per corner), and per corner a block of b^2 entries of a few operations
        nip = {3: 3, 4: 4, 8: 12}[nsh]
        f_def, f_jac = elems * nip * nsh * 40.0, elems * nip * nsh * 5.0 * b * b
        mv = nnz * b * b * 2.0
        if k == "assemble":
            what = case["what"]
            by = elem_in + (vec if what != "jacobian" else 0) + (mat + nnz * 4.0 if what != "defect" else 0)
            return {"bytes": by, "flops": (f_def if what != "jacobian" else 0) + (f_jac if what != "defect" else 0)}
        if k == "spmv":
            return {"bytes": mat + nnz * 4.0 + 2 * vec, "flops": mv}
        it = case["iters"]
        if case["solver"] == "bicgstab":
            # two products, two preconditioners and ten vector passes an iteration
            by, fl = it * (2 * (mat + nnz * 4.0) + 2 * nodes * b * b * vb + 14 * vec), it * (2 * mv + 2 * nodes * b * b * 2.0 + 20.0 * nodes * b)
        else:
            # a product, a preconditioner and the orthogonalisation against the mean basis
            q = min(it, 30) / 2.0
            by, fl = it * (mat + nnz * 4.0 + nodes * b * b * vb + (2 * q + 4) * vec), it * (mv + 8.0 * q * nodes * b)
        if k == "linear":
            return {"bytes": by, "flops": fl}
        st = case["steps"]
        return {"bytes": st * (by + 2 * elem_in + 2 * vec + mat), "flops": st * (fl + 2 * f_def + f_jac)}
    if k == "batch":
        sizes = [int(v) for v in case["sizes"].split(",")]
        n = [sizes[i % len(sizes)] for i in range(case["instances"])]
        # about 24 Newton steps of 20 Krylov steps each; a step reads the matrix hierarchy about 7 times and 8 basis vectors
        nodes = sum((v + 1) ** 2 for v in n)
        return {"bytes": 24.0 * 20 * nodes * (7 * 9 * 9 * 4 * 4 / 3 + 16 * 12), "flops": 24.0 * 20 * nodes * (7 * 9 * 9 * 2 * 4 / 3 + 16 * 6)}
    w = MLP_WIDTH
    macs = MLP_FEATURES * w + 3 * w * w + 3 * w
    if k == "predict":
        p = case["instances"] * (case["n"] + 1) ** 2
        return {"bytes": p * (8.0 + 24.0) + 4.0 * MLP_PARAMS, "flops": 2.0 * p * macs}
    p = case["slots"] * case["points"]
    # activations of four layers kept in 16 bits for the backward pass
    return {"bytes": p * (8.0 + 12.0 + 4 * 2 * 2.0 * w) + 8.0 * MLP_PARAMS, "flops": 6.0 * p * macs}


# ---- plain 64-bit results ----------------------------------------------------------

_CORNERS = {
    TRI: [[0, 0], [1, 0], [0, 1]],
    QUAD: [[0, 0], [1, 0], [1, 1], [0, 1]],
    HEX: [[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0], [0, 0, 1], [1, 0, 1], [1, 1, 1], [0, 1, 1]],
}
_EDGES = {
    TRI: [(0, 1), (1, 2), (2, 0)],
    QUAD: [(0, 1), (1, 2), (2, 3), (3, 0)],
    HEX: [(0, 1), (1, 2), (2, 3), (3, 0), (0, 4), (1, 5), (2, 6), (3, 7), (4, 5), (5, 6), (6, 7), (7, 4)],
}
_FACES = [[0, 3, 2, 1], [0, 1, 5, 4], [1, 2, 6, 5], [2, 3, 7, 6], [0, 4, 7, 3], [4, 5, 6, 7]]


def _shapes(t, xi):
    """P1 shapes [..., nsh] and local gradients [..., nsh, dim] at local points xi [..., dim]."""
    if t == TRI:
        a, b = xi[..., 0], xi[..., 1]
        g = torch.tensor([[-1.0, -1.0], [1.0, 0.0], [0.0, 1.0]], dtype=torch.float64, device=xi.device)
        return torch.stack([1 - a - b, a, b], -1), g.expand(*xi.shape[:-1], 3, 2)
    co = torch.tensor(_CORNERS[t], dtype=torch.float64, device=xi.device)
    f = co * xi[..., None, :] + (1 - co) * (1 - xi[..., None, :])  # [..., nsh, dim]
    s = 2 * co - 1
    dim = co.shape[1]
    g = [s[:, d] * torch.prod(f[..., [e for e in range(dim) if e != d]], -1) for d in range(dim)]
    return torch.prod(f, -1), torch.stack(g, -1)


def _exact_assemble(case, seed):
    t, xh, ch = _mesh(case["mesh"], case["n"])
    dev = torch.device("cuda")
    X = torch.from_numpy(xh).to(dev)
    conn = torch.from_numpy(ch.astype(np.int64)).to(dev)
    dim, nsh, ne = X.shape[1], NSH[t], conn.shape[0]
    b, P = dim + 1, dim
    U = _iterate(case, X, seed).view(-1, b)
    Uo = _iterate(case, X, seed, 0.02).view(-1, b) if case["transient"] else None
    nu, dt, rho = _nu(case), _dt(case), 1.0
    flow, lps, tr = case["stab"] == "flow", case["upwind"] == "lps", case["transient"]
    x, u = X[conn], U[conn]  # [E, nsh, dim], [E, nsh, b]
    uo = Uo[conn] if tr else None
    cen = x.mean(1)
    ref = torch.tensor(_CORNERS[t], dtype=torch.float64, device=dev)
    rcen = ref.mean(0)

    def around(p, rp, i, j):
        """edge midpoint and, in 3D, the centres of the two faces at the edge, of global or local corners p."""
        em = 0.5 * (p[..., i, :] + p[..., j, :])
        fs = [p[..., f, :].mean(-2) for f in _FACES if i in f and j in f] if dim == 3 else []
        return em, fs

    # SCV volumes
    vol = torch.empty(ne, nsh, dtype=torch.float64, device=dev)
    for a in range(nsh):
        at = [e for e in _EDGES[t] if a in e]
        q = [0.5 * (x[:, i] + x[:, j]) for i, j in at]
        if dim == 2:
            e, f = cen - x[:, a], q[0] - q[1]
            vol[:, a] = 0.5 * (e[:, 0] * f[:, 1] - e[:, 1] * f[:, 0]).abs()
        else:
            # six tetrahedra about the diagonal corner - centre: edge midpoint, face centre, edge midpoint, ...
            v = torch.zeros(ne, dtype=torch.float64, device=dev)
            for fc in _FACES:
                if a in fc:
                    fcen = x[:, fc].mean(1)
                    for (i, j), m in zip(at, q):
                        if i in fc and j in fc:
                            v += torch.linalg.det(torch.stack([m - x[:, a], fcen - x[:, a], cen - x[:, a]], 1)).abs()
            vol[:, a] = v / 6.0
    De = torch.zeros(ne, nsh, b, dtype=torch.float64, device=dev)
    want_j = case["what"] != "defect"
    Ke = torch.zeros(ne, nsh, nsh, b, b, dtype=torch.float64, device=dev) if want_j else None
    sc = dt if tr else 1.0
    for i, j in _EDGES[t]:
        em, fs = around(x, None, i, j)
        rem, rfs = around(ref, None, i, j)
        if dim == 2:
            e = cen - em
            n = torch.stack([e[:, 1], -e[:, 0]], 1)
            gip, rip = 0.5 * (em + cen), 0.5 * (rem + rcen)
        else:
            n = 0.5 * torch.linalg.cross(cen - em, fs[1] - fs[0])
            gip, rip = 0.25 * (em + cen + fs[0] + fs[1]), 0.25 * (rem + rcen + rfs[0] + rfs[1])
        n = n * torch.where(((x[:, j] - x[:, i]) * n).sum(1, keepdim=True) < 0, -1.0, 1.0)
        N, lg = _shapes(t, rip)
        J = torch.einsum("ekr,kc->erc", x, lg)
        g = torch.einsum("ecr,kc->ekr", torch.linalg.inv(J), lg)  # global gradients [E, nsh, dim]
        vel = torch.einsum("k,ekd->ed", N, u[..., :dim])
        gv = torch.einsum("ekf,ekr->efr", u, g)  # gradients of every function
        p = torch.einsum("k,ek->e", N, u[..., P])
        norm = vel.norm(dim=1)
        Vn = (vel * n).sum(1)

        def upwind(v):
            """shapes and length of the upwind of SCVF velocity v."""
            sh = torch.zeros(ne, nsh, dtype=torch.float64, device=dev)
            if case["upwind"] == "no":
                return N.expand(ne, nsh), torch.ones(ne, dtype=torch.float64, device=dev)
            if not lps:
                up = (v * n).sum(1) > 0
                sh[:, i], sh[:, j] = up.double(), (~up).double()
                return sh, torch.where(up, (gip - x[:, i]).norm(dim=1), (gip - x[:, j]).norm(dim=1))
            # the upwind ray leaves the (affine) element at the smallest parameter over its sides
            w = torch.linalg.solve(J, v)
            inf = torch.full_like(w, math.inf)
            s = torch.where(w > 0, rip / w, inf)
            if t == TRI:
                ws = w.sum(1, keepdim=True)
                s = torch.cat([s, torch.where(ws < 0, (1 - rip.sum()) / -ws, torch.full_like(ws, math.inf))], 1)
            else:
                s = torch.minimum(s, torch.where(w < 0, (1 - rip) / -w, inf))
            s = s.min(1).values
            sh, _ = _shapes(t, rip - s[:, None] * w)
            return sh, s * norm

        up, lup = upwind(vel)
        dn, ldn = upwind(-vel)
        nn = (n * n).sum(1)
        area = (0.5 * (vol[:, i] + vol[:, j])) ** 2
        ds = ((em - cen) ** 2).sum(1) if dim == 3 else nn
        nul = nu * nn / (0.5 * area + 0.375 * ds * nn)
        ncl = norm / lup
        ndl = norm / (ldn + lup) if flow else torch.zeros_like(norm)
        diag = nul + ncl + (1.0 / dt if tr else 0.0)
        upv, dnv = torch.einsum("ek,ekd->ed", up, u[..., :dim]), torch.einsum("ek,ekd->ed", dn, u[..., :dim])
        rhs = nul[:, None] * vel + ncl[:, None] * upv - gv[:, P] / rho
        if tr:
            rhs = rhs + torch.einsum("k,ekd->ed", N, uo[..., :dim]) / dt
        if flow:
            div = sum(gv[:, d, d] for d in range(dim))
            rhs = rhs + ndl[:, None] * (dnv - upv) + vel * div[:, None] - torch.einsum("edr,er->ed", gv[:, :dim], vel)
        stab = rhs / diag[:, None]
        visc = -nu * rho * (torch.einsum("edr,er->ed", gv[:, :dim], n) + torch.einsum("erd,er->ed", gv[:, :dim], n))
        flux = visc + upv * (rho * Vn)[:, None] + p[:, None] * n
        cont = rho * (stab * n).sum(1)
        full = torch.cat([flux, cont[:, None]], 1) * sc
        De[:, i] += full
        De[:, j] -= full
        if want_j:
            gn, vg = torch.einsum("ekr,er->ek", g, n), torch.einsum("ekr,er->ek", g, vel)
            B = torch.zeros(ne, nsh, b, b, dtype=torch.float64, device=dev)
            B[:, :, :dim, :dim] = -nu * rho * torch.einsum("eka,ec->ekac", g, n)
            dd = -nu * rho * gn + up * (rho * Vn)[:, None]
            for d in range(dim):
                B[:, :, d, d] += dd
            B[:, :, :dim, P] = N[None, :, None] * n[:, None, :]
            sk = nul[:, None] * N + ncl[:, None] * up
            if flow:
                sk = sk + ndl[:, None] * (dn - up) - vg
            B[:, :, P, :dim] = rho * sk[..., None] * n[:, None, :]
            if flow:
                B[:, :, P, :dim] += rho * Vn[:, None, None] * g
            B[:, :, P, P] = -gn
            B[:, :, P] /= diag[:, None, None]
            Ke[:, i] += sc * B
            Ke[:, j] -= sc * B
    if tr:
        De[..., :dim] += rho * vol[..., None] * (u - uo)[..., :dim]
        if want_j:
            for a in range(nsh):
                for d in range(dim):
                    Ke[:, a, a, d, d] += rho * vol[:, a]
    nodes = X.shape[0]
    rows, vals = _walls(case["mesh"], case["n"]) if case["walls"] else (np.zeros(0, np.int32), np.zeros(0))
    rows = torch.from_numpy(rows.astype(np.int64)).to(dev)
    D = torch.zeros(nodes, b, dtype=torch.float64, device=dev).index_add_(0, conn.reshape(-1), De.reshape(-1, b)).reshape(-1)
    D[rows] = U.reshape(-1)[rows] - torch.from_numpy(vals).to(dev)
    if not want_j:
        return [D]
    keys = (conn[:, :, None] * nodes + conn[:, None, :]).reshape(-1)
    blocks, at = torch.unique(keys, return_inverse=True)
    A = torch.zeros(blocks.numel(), b * b, dtype=torch.float64, device=dev)
    A.index_add_(0, at, Ke.reshape(-1, b * b))
    A = A.view(-1, b, b)
    wall = torch.zeros(nodes * b, dtype=torch.bool, device=dev)
    wall[rows] = True
    brow, bcol = blocks // nodes, blocks % nodes
    for f in range(b):
        hit = wall[brow * b + f]
        A[hit, f, :] = 0.0
        A[hit & (brow == bcol), f, f] = 1.0
    A = A.reshape(-1)
    return [D, A] if case["what"] == "both" else [A]


def _exact_spmv(case, seed):
    t, xh, ch = _mesh(case["mesh"], case["n"])
    b = xh.shape[1] + 1
    conn = torch.from_numpy(ch.astype(np.int64)).cuda()
    n = xh.shape[0]
    blocks = torch.unique((conn[:, :, None] * n + conn[:, None, :]).reshape(-1))
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    a = torch.randn(blocks.numel() * b * b, generator=g, dtype=_dtype(case), device="cuda").double().view(-1, b, b)
    x = torch.randn(n * b, generator=g, dtype=torch.float64, device="cuda").view(-1, b)
    p = torch.einsum("qij,qj->qi", a, x[blocks % n])
    return [torch.zeros(n, b, dtype=torch.float64, device="cuda").index_add_(0, blocks // n, p).reshape(-1)]


def _params(seed):
    """The network's parameters of a seed (the flat layout of get_params): He-uniform weights, small FiLM maps."""
    r = np.random.RandomState(seed)
    parts = []
    for layer in range(4):
        k = MLP_FEATURES if layer == 0 else MLP_WIDTH
        parts.append(r.uniform(-1, 1, MLP_WIDTH * k) * math.sqrt(6.0 / k))
        for m in (1, 2, 1, 2, 1):
            parts.append(r.uniform(-0.1, 0.1, m * MLP_WIDTH))
    parts += [r.uniform(-1, 1, 3 * MLP_WIDTH) * math.sqrt(3.0 / MLP_WIDTH), r.uniform(-0.1, 0.1, 3)]
    return np.concatenate(parts).astype(np.float32)


def _exact_net(p, xy, cond, per):
    """The network's output [n, 3] at xy, slot s holding points [s * per, (s + 1) * per)."""
    w, at = MLP_WIDTH, [0]

    def take(*shape):
        k = math.prod(shape)
        at[0] += k
        return p[at[0] - k: at[0]].reshape(shape)

    k = torch.arange(1, 17, dtype=torch.float64, device=xy.device)
    ax, ay = xy[:, :1] * k * math.pi, xy[:, 1:] * k * math.pi
    h = torch.stack([torch.sin(ax), torch.cos(ax), torch.sin(ay), torch.cos(ay)], -1).reshape(xy.shape[0], -1)
    for _ in range(4):
        W, b, Gw, Gb, Bw, Bb = take(w, h.shape[1]), take(w), take(w, 2), take(w), take(w, 2), take(w)
        ga, be = 1 + cond @ Gw.T + Gb, cond @ Bw.T + Bb
        z = ga.repeat_interleave(per, 0) * (h @ W.T + b) + be.repeat_interleave(per, 0)
        h = z * torch.sigmoid(z)
    Wh, bh = take(3, w), take(3)
    return h @ Wh.T + bh


def exact(case, seed):
    k = case["kind"]
    if k == "assemble":
        return _exact_assemble(case, seed)
    if k == "spmv":
        return _exact_spmv(case, seed)
    if k in ("linear", "newton", "batch"):
        return None  # a bounded number of Krylov steps has no plain value of its own
    p = torch.from_numpy(_params(seed)).double().cuda()
    if k == "predict":
        r = np.random.RandomState(seed)
        n, nn = case["instances"], (case["n"] + 1) ** 2
        xy = torch.from_numpy(mesh.structured_quads(case["n"])[1].astype(np.float32)).double().cuda().repeat(n, 1)
        cond = torch.from_numpy(r.uniform(-1, 1, size=(n, 2)).astype(np.float32)).double().cuda()
        lid = torch.from_numpy(r.uniform(0.5, 2.0, size=n).astype(np.float32)).double().cuda().repeat_interleave(nn)[:, None]
        out = _exact_net(p, xy, cond, nn)
        return [torch.cat([lid * out[:, :2], lid * lid * out[:, 2:]], 1).reshape(-1)]
    n = case["slots"] * case["points"]
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    xy = torch.rand(n, 2, generator=g, dtype=torch.float32, device="cuda").double()
    target = torch.randn(n, 3, generator=g, dtype=torch.float32, device="cuda") * 0.3
    target = target.double()
    cond = torch.from_numpy(np.random.RandomState(seed).uniform(-1, 1, size=(case["slots"], 2)).astype(np.float32)).double().cuda()
    p.requires_grad_(True)
    loss = ((_exact_net(p, xy, cond, case["points"]) - target) ** 2).mean()
    loss.backward()
    return [float(loss), p.grad]
