"""The restarted GMRES where a block has several tiles and the last block sums many partials: more
than 304 x 256 unknowns with a remainder tile, and 32 < blocks < 304; restart lengths 30 (two
cycles) and 64. Against the same algorithm in float64 on the assembled sparse matrix."""
import numpy as np
import pytest
import scipy.sparse

from plugin_navierstokes_gb300 import NavierStokesFV1, mesh
from test_gpu_gmres import reference

pytestmark = pytest.mark.gpu

# (mesh, cells, restart, iterations, least blocks, tiles of a block)
CASES = [("quad", 100, 30, 45, 33, 1), ("quad", 165, 30, 45, 304, 2), ("quad", 165, 64, 66, 304, 2), ("hex", 30, 30, 40, 304, 2), ("tri", 240, 30, 33, 304, 3)]


def sparse(rp, ci, v, b):
    """CSR matrix of b x b blocks v."""
    return scipy.sparse.bsr_matrix((v, ci, rp), shape=((rp.size - 1) * b,) * 2).tocsr()


@pytest.mark.parametrize("kind,n,m,iters,blocks,tiles", CASES)
def test_gmres_matches_reference(cuda, kind, n, m, iters, blocks, tiles):
    import torch

    t, x, c = {"quad": mesh.structured_quads, "tri": mesh.jittered_triangles, "hex": mesh.structured_hexes}[kind](n)
    b = x.shape[1] + 1
    d = NavierStokesFV1(dim=b - 1)
    d.set_kinematic_viscosity(0.01)
    d.set_upwind("full")
    d.set_stabilization("flow")
    d.set_mesh(t, x, c)
    d.set_dirichlet(*mesh.cavity_dirichlet(x))
    size = x.shape[0] * b
    grid = min(304, -(-size // 256))
    per = -(-(-(-size // grid)) // 32) * 32
    assert grid >= blocks and -(-per // 256) == tiles
    u = torch.from_numpy(0.3 * (2 * mesh.uniform(3, size) - 1)).to(cuda)
    rp, ci = d.pattern()
    vals = torch.empty(ci.size * b * b, dtype=torch.float64, device=cuda)
    d.assemble_jacobian(u, vals)
    v = vals.cpu().numpy().reshape(-1, b, b)
    Dinv = np.linalg.inv(v[np.repeat(np.arange(rp.size - 1), np.diff(rp)) == ci])
    A = sparse(rp, ci, v, b)
    rhs = 2 * mesh.uniform(7, size) - 1
    sol = torch.empty(size, dtype=torch.float64, device=cuda)
    r = d.linear_solve(vals, torch.from_numpy(rhs).to(cuda), sol, lin_rtol=1e-13, lin_max_iter=iters, linear_solver="gmres", gmres_restart=m,
                       raise_on_error=False)
    assert r["iterations"] == iters
    got, ref = sol.cpu().numpy(), reference(A, Dinv, rhs, m, iters)
    # backward stable: rounding of sums of this length (about 1e-14) times the condition of the
    # preconditioned operator on the Krylov space (below 50 here)
    assert np.linalg.norm(got - ref) <= 1e-10 * np.linalg.norm(ref)
    true = np.linalg.norm(rhs - A @ got) / np.linalg.norm(rhs)
    assert abs(r["relres"] - true) <= 1e-12
