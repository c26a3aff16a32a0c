"""The one-launch FP32 Jacobian of 2D meshes: the same bits as colour by colour (which instances
that are skipped, a mesh with an edge in three elements and the oracle's tolerance stand
for), small and shuffled meshes, a node with many triangles, both entry points, repeated runs."""
import numpy as np
import pytest

import oracle
from _cases import rel_err
from plugin_navierstokes_gb300 import NavierStokesFV1, mesh

pytestmark = pytest.mark.gpu
TOL32 = 2e-5


def fan(n):
    """n triangles around one node."""
    a = 2 * np.pi * np.arange(n) / n
    x = np.concatenate([[[0.0, 0.0]], np.stack([np.cos(a), np.sin(a)], 1)])
    k = np.arange(n)
    return 2, x, np.stack([np.zeros(n, int), 1 + k, 1 + (k + 1) % n], 1).astype(np.int32)


def make(name):
    if name == "fan":
        return fan(40)
    if name == "book":   # an edge in three triangles: colour by colour
        return 2, np.array([[0, 0], [1, 0], [0.4, 1], [0.5, -1], [0.6, 0.7]], float), np.array([[0, 1, 2], [1, 0, 3], [0, 1, 4]], np.int32)
    if name == "collapsed":   # quadrilaterals with a node twice
        t, x, c = mesh.structured_quads(4)
        c = c.copy()
        c[5, 2] = c[5, 1]
        c[10, 3] = c[10, 2]
        return t, x, c
    base, n = name.split()
    t, x, c = {"tri": mesh.jittered_triangles, "quad": mesh.structured_quads}[base](int(n.rstrip("s")))
    if n.endswith("s"):
        p = np.argsort(mesh.uniform(8, x.shape[0]))
        x, c = np.ascontiguousarray(x[np.argsort(p)]), p[c].astype(np.int32)
    return t, x, c


@pytest.mark.parametrize("name", ["tri 1", "tri 9", "tri 40", "tri 23s", "fan", "book", "collapsed", "quad 1", "quad 12", "quad 17s"])
@pytest.mark.parametrize("transient", [False, True])
def test_matches_oracle_and_itself(cuda, name, transient):
    import torch

    t, x, c = make(name)
    discs = (NavierStokesFV1(dim=2), oracle.Oracle(2))
    for d in discs:
        d.set_kinematic_viscosity(0.02)
        d.set_upwind("full")
        d.set_stabilization("flow")
        d.set_density(1.3)
        d.set_mesh(t, x, c)
    d, o = discs
    U = 2 * mesh.uniform(11, x.shape[0] * 3) - 1
    Uo, dt = (0.9 * U, 0.05) if transient else (None, 0.0)
    _, Jref = o.assemble(U.reshape(-1, 3), None if Uo is None else Uo.reshape(-1, 3), dt)
    tu = torch.from_numpy(U).to(cuda)
    tuo = None if Uo is None else torch.from_numpy(Uo).to(cuda)
    J = [torch.full((Jref.size,), float("nan"), dtype=torch.float32, device=cuda) for _ in range(3)]
    d.assemble_jacobian(tu, J[0], tuo, dt)
    d.assemble_defect_jacobian(tu, torch.empty_like(tu), J[1], tuo, dt)
    d.assemble_jacobian(tu, J[2], tuo, dt)
    assert rel_err(J[0].double().cpu().numpy().reshape(Jref.shape), Jref) <= TOL32
    assert torch.equal(J[0], J[1]) and torch.equal(J[0], J[2])


@pytest.mark.parametrize("name", ["tri 23s", "quad 12"])
def test_same_bits_as_colour_by_colour(cuda, name):
    """A third triangle far away on a shared pair of nodes sends the whole mesh colour by colour: the
    rows that it does not touch keep their bits."""
    import torch

    t, x, c = make(name)
    values = []
    for extra in (False, True):
        X, C = x, c
        if extra:
            # three more elements that share one edge, disjoint from the mesh
            k = x.shape[0]
            tail = np.array([[5, 5], [6, 5], [5.4, 6], [5.5, 4], [5.6, 5.7]], float)
            add = np.array([[0, 1, 2], [1, 0, 3], [0, 1, 4]])
            if t == 3:
                tail = np.concatenate([tail, [[6.1, 6], [6.2, 4], [6.3, 5.8]]])
                add = np.array([[0, 1, 5, 2], [1, 0, 3, 6], [0, 1, 7, 4]])
            X, C = np.concatenate([x, tail]), np.concatenate([c, (add + k).astype(np.int32)])
        d = NavierStokesFV1(dim=2)
        d.set_kinematic_viscosity(0.02)
        d.set_upwind("lps")
        d.set_stabilization("fields")
        d.set_mesh(t, np.ascontiguousarray(X), C)
        U = np.zeros(X.shape[0] * 3)
        U[: x.shape[0] * 3] = 2 * mesh.uniform(11, x.shape[0] * 3) - 1
        U[x.shape[0] * 3:] = 0.1
        rp, _ = d.pattern()
        J = torch.empty(d.pattern_info()["nnz_blocks"] * 9, dtype=torch.float32, device=cuda)
        d.assemble_jacobian(torch.from_numpy(U).to(cuda), J)
        values.append(J[: rp[x.shape[0]] * 9].clone())
    assert torch.equal(values[0], values[1])
