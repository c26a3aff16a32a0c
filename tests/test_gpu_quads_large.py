"""Quadrilaterals on both sides of the lane split (4 x 152 x 8 = 4,864 elements of a launch, affine and
general elements being launches of their own), the two-directions-per-lane kernels among
them: against the oracle, the defect and the Jacobian alone, and a second run for equal bits.
Left-handed general elements too: their normal has a sign of its own."""
import numpy as np
import pytest

import oracle
from _cases import rel_err
from plugin_navierstokes_gb300 import NavierStokesFV1, mesh
from test_gpu_fast_assembly import TOL64, make

pytestmark = pytest.mark.gpu
SPLIT_LIMIT = 4 * 152 * 8

# (mesh, cells, elements of a launch above the limit)
MESHES = [("quad", 138, False), ("quad", 142, True), ("quad-j", 138, False), ("quad-j", 142, True), ("quad-m", 204, True), ("quad-jl", 145, True)]


def affine(x, c):
    p = x[c]
    dev = np.abs((p[:, 2] - p[:, 1]) - (p[:, 3] - p[:, 0])).max(1)
    return dev <= 1e-14 * np.maximum(np.abs(p[:, 1] - p[:, 0]), np.abs(p[:, 3] - p[:, 0])).max(1)


@pytest.mark.parametrize("upwind,stab,transient", [("full", "flow", False), ("full", "fields", True), ("lps", "flow", True), ("lps", "fields", False), ("no", "flow", True)])
@pytest.mark.parametrize("kind,n,above", MESHES)
def test_matches_oracle(cuda, kind, n, above, upwind, stab, transient):
    check(cuda, kind, n, upwind, stab, transient, above)


@pytest.mark.parametrize("upwind", ["full", "lps", "no"])
@pytest.mark.parametrize("stab", ["flow", "fields"])
@pytest.mark.parametrize("kind,n", [("quad-jl", 1), ("quad-jl", 9), ("quad-ml", 8), ("hex-jl", 1), ("hex-jl", 4), ("hex-ml", 4), ("tri-jl", 5)])
def test_left_handed_general_elements(cuda, kind, n, stab, upwind):
    check(cuda, kind, n, upwind, stab, n % 2 == 1, None)


def check(cuda, kind, n, upwind, stab, transient, above):
    import torch

    t, x, c = make(kind, n)
    dim = x.shape[1]
    b = dim + 1
    discs = (NavierStokesFV1(dim=dim), oracle.Oracle(dim))
    for d in discs:
        d.set_kinematic_viscosity(0.02)
        d.set_upwind(upwind)
        d.set_stabilization(stab)
        d.set_source([0.3, -0.2, 0.1][:dim])
        d.set_mesh(t, x, c)
    d, o = discs
    if above is not None:
        # every launch of the general kernels is on the intended side (LPS: the affine ones)
        colour, aff = d.coloring(), affine(x, c)
        counts = [np.bincount(colour[part]) for part in (aff, ~aff) if part.any()]
        assert len(counts) == (2 if "m" in kind else 1)
        assert all((v > SPLIT_LIMIT).all() == above and (v <= SPLIT_LIMIT).all() != above for v in counts)
    U = 2 * mesh.uniform(13, x.shape[0] * b).reshape(-1, b) - 1
    Uo, dt = (0.8 * U, 0.03) if transient else (None, 0.0)
    Dref, Jref = o.assemble(U, Uo, dt)
    tu = torch.from_numpy(U.ravel()).to(cuda)
    tuo = None if Uo is None else torch.from_numpy(Uo.ravel()).to(cuda)
    D, J = torch.full_like(tu, float("nan")), torch.full((Jref.size,), float("nan"), dtype=torch.float64, device=cuda)
    D2, J2 = torch.full_like(D, float("nan")), torch.full_like(J, float("nan"))
    d.assemble_defect(tu, D2, tuo, dt)
    d.assemble_jacobian(tu, J2, tuo, dt)
    d.assemble_defect_jacobian(tu, D, J, tuo, dt)
    for got, ref in ((D, Dref), (D2, Dref), (J, Jref), (J2, Jref)):
        assert rel_err(got.cpu().numpy().reshape(ref.shape), ref) <= TOL64
    d.assemble_defect_jacobian(tu, D2, J2, tuo, dt)
    assert torch.equal(D, D2) and torch.equal(J, J2), "not the same bits"
