"""The staged diagonal blocks of the one-launch FP32 Jacobian take device memory from the first FP32
Jacobian of a 2D mesh on, and give it back where a workspace does not fit otherwise."""
import pytest

from plugin_navierstokes_gb300 import NavierStokesFV1, mesh

pytestmark = pytest.mark.gpu
MB = 1 << 20


def disc(n):
    import torch

    t, x, c = mesh.structured_quads(n)
    d = NavierStokesFV1(dim=2)
    d.set_kinematic_viscosity(0.02)
    d.set_upwind("full")
    d.set_stabilization("flow")
    u = torch.from_numpy(2 * mesh.uniform(3, x.shape[0] * 3) - 1).cuda()
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    d.set_mesh(t, x, c)
    return d, u, x, c, free0


def test_memory_from_the_first_fp32_jacobian_on(cuda):
    import torch

    used = lambda: free0 - torch.cuda.mem_get_info()[0]
    # loads the kernels first: their code takes device memory too
    d, u, _, _, _ = disc(4)
    J = [torch.empty(d.pattern_info()["nnz_blocks"] * 9, dtype=t, device=cuda) for t in (torch.float64, torch.float32)]
    for v in J:
        d.assemble_jacobian(u, v)
    n = 500
    J = [torch.empty((3 * n + 1) ** 2 * 9, dtype=t, device=cuda) for t in (torch.float64, torch.float32)]
    d, u, x, c, free0 = disc(n)
    nnz = d.pattern_info()["nnz_blocks"]
    # coordinates, connectivity, block indices, colours, row pointers, columns, diagonal positions;
    # an allocation is rounded up by at most 2 MB
    mesh_bytes = x.nbytes + c.nbytes + 4 * (16 * c.shape[0] + c.shape[0] + 2 * x.shape[0] + nnz)
    stage = 36 * c.size
    assert stage > 30 * MB
    d.assemble_jacobian(u, J[0])
    assert used() <= mesh_bytes + 16 * MB
    d.assemble_jacobian(u, J[1])
    assert used() >= mesh_bytes + stage
    assert float((J[0] - J[1].double()).abs().max()) <= 2e-5 * float(J[0].abs().max())


def test_staging_is_given_back_for_a_workspace(cuda):
    """A solve whose workspace fits only without the staging still runs; the Jacobian keeps its bits."""
    import torch

    def solve(d, J, rhs, x):
        return d.linear_solve(J, rhs, x, lin_rtol=1e-12, lin_max_iter=3, linear_solver="gmres", gmres_restart=64, raise_on_error=False)

    out = []
    for n, short in ((4, False), (800, True)):   # the small one loads the kernels
        d, u, x, c, _ = disc(n)
        d.set_dirichlet(*mesh.cavity_dirichlet(x))
        J = torch.empty(d.pattern_info()["nnz_blocks"] * 9, dtype=torch.float32, device=cuda)
        d.assemble_jacobian(u, J)
        rhs, sol = torch.ones_like(u), torch.empty_like(u)
        if not short:
            solve(d, J, rhs, sol)
            continue
        again = torch.empty_like(J)
        torch.cuda.empty_cache()
        # Krylov vectors, matrix and inverse blocks, four vectors of the Newton loop
        work = (10 + 2 * 65 + 4) * u.numel() * 8 + J.numel() * 4 + u.numel() * 12
        stage = 36 * c.size
        ballast = torch.empty(torch.cuda.mem_get_info()[0] - work + 20 * MB, dtype=torch.uint8, device=cuda)
        assert stage > 80 * MB and torch.cuda.mem_get_info()[0] < work
        try:
            r = solve(d, J, rhs, sol)
            assert r["iterations"] == 3, (r, d.last_error())
            d.assemble_jacobian(u, again)   # colour by colour now
            assert torch.equal(J, again)
        finally:
            del ballast
            torch.cuda.empty_cache()
