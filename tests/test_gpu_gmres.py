"""The device-resident restarted GMRES against the same algorithm in float64 numpy on the
assembled matrix: meshes below and above one 256-entry tile, restart lengths 1 to 64, a
remainder in the last warp of basis vectors, several cycles and both matrix precisions."""
import numpy as np
import pytest

from plugin_navierstokes_gb300 import NavierStokesFV1, mesh

pytestmark = pytest.mark.gpu

# (mesh, cells, restart, iterations)
CASES = [("quad", 3, 64, 30), ("quad", 8, 1, 6), ("quad", 9, 7, 20), ("tri", 17, 30, 45), ("hex", 4, 9, 25), ("quad", 21, 64, 64), ("hex", 2, 8, 16)]


def reference(A, Dinv, rhs, m, maxit):
    """x after maxit iterations of GMRES(m), right preconditioned, two Gram-Schmidt passes."""
    n, b = rhs.size, Dinv.shape[1]
    prec = lambda v: np.einsum("rij,rj->ri", Dinv, v.reshape(-1, b)).ravel()
    x, it = np.zeros(n), 0
    while it < maxit:
        r = rhs - A @ x
        beta = np.linalg.norm(r)
        V, Z, H, j = [r / beta], [], np.zeros((m + 1, m)), 0
        while j < m and it < maxit:
            Z.append(prec(V[j]))
            w = A @ Z[j]
            B = np.array(V)
            for _ in range(2):
                h = B @ w
                w = w - B.T @ h
                H[: j + 1, j] += h
            H[j + 1, j] = np.linalg.norm(w)
            V.append(w / H[j + 1, j])
            j, it = j + 1, it + 1
        e = np.zeros(j + 1)
        e[0] = beta
        x = x + np.array(Z).T @ np.linalg.lstsq(H[: j + 1, :j], e, rcond=None)[0]
    return x


def system(kind, n, prec):
    import torch

    t, x, c = {"quad": mesh.structured_quads, "tri": mesh.jittered_triangles, "hex": mesh.structured_hexes}[kind](n)
    dim = x.shape[1]
    d = NavierStokesFV1("u,v,w,p" if dim == 3 else "u,v,p", "Inner")
    d.set_kinematic_viscosity(0.01)
    d.set_upwind("full")
    d.set_stabilization("flow")
    d.set_mesh(t, x, c)
    d.set_dirichlet(*mesh.cavity_dirichlet(x))
    b = dim + 1
    u = torch.from_numpy(0.3 * (2 * mesh.uniform(3, x.shape[0] * b) - 1)).cuda()
    rp, ci = d.pattern()
    vals = torch.empty(ci.size * b * b, dtype=torch.float64 if prec == "f64" else torch.float32, device="cuda")
    d.assemble_jacobian(u, vals)
    v = vals.double().cpu().numpy().reshape(-1, b, b)
    A = np.zeros((x.shape[0], b, x.shape[0], b))
    row = np.repeat(np.arange(x.shape[0]), np.diff(rp))
    A[row, :, ci, :] = v
    Dinv = np.linalg.inv(v[row == ci])
    if prec == "f32":
        Dinv = Dinv.astype(np.float32).astype(np.float64)
    return d, vals, A.reshape(x.shape[0] * b, -1), Dinv, b


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("kind,n,m,iters", CASES)
def test_gmres_matches_reference(kind, n, m, iters, prec):
    import torch

    d, vals, A, Dinv, b = system(kind, n, prec)
    rhs = 2 * mesh.uniform(7, A.shape[0]) - 1
    x = torch.empty(rhs.size, dtype=torch.float64, device="cuda")
    r = d.linear_solve(vals, torch.from_numpy(rhs).cuda(), x, lin_rtol=1e-13, lin_max_iter=iters, linear_solver="gmres", gmres_restart=m,
                       raise_on_error=False)
    # the Krylov space of the smallest meshes is exhausted before the limit: then it has converged
    assert r["iterations"] == iters or (r["iterations"] < iters and r["relres"] < 1e-13)
    got, ref = x.cpu().numpy(), reference(A, Dinv, rhs, m, r["iterations"])
    # FP32 matrices: the product is accurate to about 1e-13 and a few inverse entries may round
    # the other way (6e-8); GMRES is backward stable, so both enter x times the condition of the
    # least-squares problem (below 1e2 on these systems)
    assert np.linalg.norm(got - ref) <= (1e-9 if prec == "f64" else 1e-5) * np.linalg.norm(ref)
    # the reported estimate is the residual of the returned x
    true = np.linalg.norm(rhs - A @ got) / np.linalg.norm(rhs)
    assert abs(r["relres"] - true) <= 1e-9


def test_gmres_stops():
    """Tolerance reached inside a cycle, a zero right-hand side, and a non-finite one."""
    import torch

    d, vals, A, Dinv, b = system("quad", 6, "f64")
    n = A.shape[0]
    rhs = 2 * mesh.uniform(8, n) - 1
    x = torch.full((n,), 7.0, dtype=torch.float64, device="cuda")
    r = d.linear_solve(vals, torch.from_numpy(rhs).cuda(), x, lin_rtol=1e-8, lin_max_iter=500, linear_solver="gmres", gmres_restart=64)
    assert r["status"] == 0 and r["relres"] < 1e-8
    assert np.linalg.norm(rhs - A @ x.cpu().numpy()) <= 1.01e-8 * np.linalg.norm(rhs)
    x.fill_(7.0)
    r = d.linear_solve(vals, torch.zeros(n, dtype=torch.float64, device="cuda"), x, linear_solver="gmres", raise_on_error=False)
    assert r["iterations"] == 0 and float(x.abs().max()) == 0.0
    bad = torch.from_numpy(rhs).cuda()
    bad[3] = float("nan")
    r = d.linear_solve(vals, bad, x, linear_solver="gmres", raise_on_error=False)
    assert r["status"] == 5
