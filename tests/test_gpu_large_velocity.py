"""A velocity whose square overflows (1e160 at one node): the Jacobian entries that are finite with the
oracle's square root are finite here, with the same values, and the others are not."""
import numpy as np
import pytest

import oracle
from plugin_navierstokes_gb300 import NavierStokesFV1, mesh
from test_gpu_fast_assembly import TOL64, make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("upwind", ["full", "no"])
@pytest.mark.parametrize("stab", ["flow", "fields"])
@pytest.mark.parametrize("kind,n", [("tri", 6), ("tet", 2), ("quad", 5), ("quad-j", 5), ("hex", 3), ("hex-j", 3)])
def test_finite_entries_stay_finite(cuda, kind, n, stab, upwind):
    import torch

    t, x, c = make(kind, n)
    b = x.shape[1] + 1
    discs = (NavierStokesFV1(dim=b - 1), oracle.Oracle(b - 1))
    for d in discs:
        d.set_kinematic_viscosity(0.02)
        d.set_upwind(upwind)
        d.set_stabilization(stab)
        d.set_mesh(t, x, c)
    U = (2 * mesh.uniform(11, x.shape[0] * b) - 1).reshape(-1, b)
    U[x.shape[0] // 2, 0] = 1e160
    with np.errstate(all="ignore"):
        ref = discs[1].assemble(U)
    u = torch.from_numpy(U.ravel()).to(cuda)
    D, J = torch.empty_like(u), torch.empty(ref[1].size, dtype=torch.float64, device=cuda)
    discs[0].assemble_defect_jacobian(u, D, J)
    got, want = J.cpu().numpy().ravel(), np.asarray(ref[1]).ravel()
    fin = np.isfinite(want)
    assert not fin.all() and np.array_equal(np.isfinite(got), fin)
    # the pressure column of the pressure rows: no velocity enters its terms but through the diagonal
    # factor, which is 0 at the overflow (other entries lose what cancels against 1e160)
    p = slice(b * b - 1, None, b * b)
    assert fin[p].all() and np.abs(got[p] - want[p]).max() <= TOL64 * np.abs(want[p]).max()
