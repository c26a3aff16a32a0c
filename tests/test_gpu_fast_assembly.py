"""The specialised FP64 assembly kernels against the oracle: element counts below, at and above a
warp's share, affine, distorted and mixed meshes, left- and right-handed elements, every
upwind x stabilisation they serve and the options that enter them; and that a second run
gives the same bits. Tolerance as in test_gpu_assembly.py (FP64 rounding of the same terms)."""
import numpy as np
import pytest

import oracle
from _cases import rel_err
from plugin_navierstokes_gb300 import NavierStokesFV1, mesh

pytestmark = pytest.mark.gpu
TOL64 = 1e-12


def make(kind, n):
    """kind: base mesh, then s(heared: affine but not axis-aligned), j(ittered), m(ixed), l(eft-handed)."""
    base, mods = kind.split("-") if "-" in kind else (kind, "")
    t, x, c = {"quad": mesh.structured_quads, "hex": mesh.structured_hexes, "tri": mesh.jittered_triangles, "tet": tets}[base](n)
    x = x.copy()
    dim = x.shape[1]
    if "j" in mods or "m" in mods:
        move = (2 * mesh.uniform(5, x.size).reshape(x.shape) - 1) * 0.12 / n
        if "m" in mods:
            move[x[:, 0] < 0.5] = 0.0
        x = x + move
    if "s" in mods:
        a = np.eye(dim) + 0.3 * (mesh.uniform(6, dim * dim).reshape(dim, dim) - 0.5)
        x = x @ a.T
    if "l" in mods:
        x[:, 0] = -x[:, 0]
    return t, np.ascontiguousarray(x), c


def tets(n):
    """Each hexahedron as six tetrahedra around a diagonal."""
    _, x, c = mesh.structured_hexes(n)
    six = [(0, 1, 2, 6), (0, 2, 3, 6), (0, 3, 7, 6), (0, 7, 4, 6), (0, 4, 5, 6), (0, 5, 1, 6)]
    x = x + (2 * mesh.uniform(9, x.size).reshape(x.shape) - 1) * 0.1 / n
    return 4, x, np.concatenate([c[:, s] for s in six]).astype(np.int32)


KINDS = ["quad", "quad-s", "quad-j", "quad-m", "quad-l", "hex", "hex-s", "hex-j", "hex-m", "hex-l", "tri", "tri-l", "tet", "tet-l"]
SIZES = {"quad": [1, 4, 9, 23], "hex": [1, 2, 5], "tri": [1, 3, 17], "tet": [1, 3]}


@pytest.mark.parametrize("upwind", ["full", "lps", "no"])
@pytest.mark.parametrize("stab", ["flow", "fields"])
@pytest.mark.parametrize("kind", KINDS)
def test_matches_oracle(cuda, kind, stab, upwind):
    import torch

    for k, n in enumerate(SIZES[kind.split("-")[0]]):
        t, x, c = make(kind, n)
        dim = x.shape[1]
        b = dim + 1
        transient, options = k % 2 == 0, k != 1
        discs = (NavierStokesFV1(dim=dim), oracle.Oracle(dim))
        for d in discs:
            d.set_kinematic_viscosity(0.02)
            d.set_upwind(upwind)
            d.set_stabilization(stab)
            if options:
                d.set_density(1.7)
                d.set_source([0.3, -0.2, 0.1][:dim])
            d.set_mesh(t, x, c)
        d, o = discs
        U = 2 * mesh.uniform(11 + k, x.shape[0] * b).reshape(-1, b) - 1
        if k == 0:
            U[: x.shape[0] // 2, :dim] = 0.0   # integration points without a velocity
        Uo = 0.8 * U if transient else None
        dt = 0.03 if transient else 0.0
        Dref, Jref = o.assemble(U, Uo, dt)
        tu = torch.from_numpy(U.ravel()).to(cuda)
        tuo = None if Uo is None else torch.from_numpy(Uo.ravel()).to(cuda)
        nan = lambda m: torch.full((m,), float("nan"), dtype=torch.float64, device=cuda)
        D, D2, D3, J, J2 = nan(Dref.size), nan(Dref.size), nan(Dref.size), nan(Jref.size), nan(Jref.size)
        d.assemble_defect_jacobian(tu, D, J, tuo, dt)
        d.assemble_defect(tu, D2, tuo, dt)
        d.assemble_jacobian(tu, J2, tuo, dt)
        for got, ref in ((D, Dref), (D2, Dref), (J, Jref), (J2, Jref)):
            assert rel_err(got.cpu().numpy().reshape(ref.shape), ref) <= TOL64, (kind, n)
        for threads in (32, 96):
            d.set_assembly_threads(threads)
            d.assemble_defect_jacobian(tu, D3, J2, tuo, dt)
            assert torch.equal(D, D3) and torch.equal(J, J2), "not the same bits"


@pytest.mark.parametrize("n", [68, 142])
def test_quads_around_the_lane_split(cuda, n):
    """Colours just below and above the element count at which a lane takes both directions again."""
    import torch

    t, x, c = make("quad-m", n)
    discs = (NavierStokesFV1(dim=2), oracle.Oracle(2))
    for d in discs:
        d.set_kinematic_viscosity(0.02)
        d.set_upwind("full")
        d.set_stabilization("flow")
        d.set_mesh(t, x, c)
    U = 2 * mesh.uniform(3, x.shape[0] * 3) - 1
    Dref, Jref = discs[1].assemble(U.reshape(-1, 3))
    u = torch.from_numpy(U).to(cuda)
    D, J = torch.empty_like(u), torch.empty(Jref.size, dtype=torch.float64, device=cuda)
    discs[0].assemble_defect_jacobian(u, D, J)
    assert rel_err(D.cpu().numpy().reshape(Dref.shape), Dref) <= TOL64
    assert rel_err(J.cpu().numpy().reshape(Jref.shape), Jref) <= TOL64


@pytest.mark.parametrize("kind,n", [("quad", 6), ("hex-j", 3), ("tri", 6)])
def test_elem_viscosity_and_zero_state(cuda, kind, n):
    """Per-element viscosity, and the state at rest (every upwind ties)."""
    import torch

    t, x, c = make(kind, n)
    dim = x.shape[1]
    nu = 0.01 + 0.05 * mesh.uniform(3, c.shape[0])
    # the oracle has one viscosity: its element contributions are summed here
    U = 2 * mesh.uniform(4, x.shape[0] * (dim + 1)) - 1
    for state in (U, np.zeros_like(U)):
        d = NavierStokesFV1(dim=dim)
        d.set_kinematic_viscosity(1.0)
        d.set_upwind("full")
        d.set_stabilization("flow")
        d.set_mesh(t, x, c)
        d.set_elem_viscosity(nu)
        u = torch.from_numpy(state).to(cuda)
        D = torch.empty_like(u)
        d.assemble_defect(u, D)
        ref = np.zeros((x.shape[0], dim + 1))
        for e in range(c.shape[0]):
            o = oracle.Oracle(dim)
            o.set_kinematic_viscosity(nu[e])
            o.set_upwind("full")
            o.set_stabilization("flow")
            loc = state.reshape(-1, dim + 1)[c[e]].T.ravel()[None]
            r = o.elem_batch(t, x[c[e]][None], loc, want=("defA",))["defA"].reshape(dim + 1, -1)
            np.add.at(ref, c[e], r.T)
        assert np.abs(D.cpu().numpy().reshape(ref.shape) - ref).max() <= TOL64 * max(np.abs(ref).max(), 1e-300)


def test_not_a_number_is_reported(cuda):
    """LPS finds no side for a velocity that is not a number, as the general path."""
    import torch
    from plugin_navierstokes_gb300 import NSFV1Error

    for kind in ("quad", "hex", "tri"):
        t, x, c = make(kind, 2)
        d = NavierStokesFV1(dim=x.shape[1])
        d.set_kinematic_viscosity(0.01)
        d.set_upwind("lps")
        d.set_stabilization("flow")
        d.set_mesh(t, x, c)
        u = torch.full((x.size + x.shape[0],), float("nan"), dtype=torch.float64, device=cuda)
        with pytest.raises(NSFV1Error, match="cut side"):
            d.assemble_defect(u, torch.empty_like(u))
