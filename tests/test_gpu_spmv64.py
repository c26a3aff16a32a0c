"""The FP64 block product of 3D patterns (16 lanes per row) against float64 numpy: rows of fewer
blocks than one unrolled trip (a single hexahedron: 8), of exactly 27, remainders in between
(tetrahedra, prisms), row counts that do not fill a CTA, and values that overflow if a lane
reads another block. Tolerance: the rounding of one sum, 4e-16 sum |a x| per 8 terms."""
import numpy as np
import pytest

from plugin_navierstokes_gb300 import NavierStokesFV1, mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n", [("hex", 1), ("hex", 2), ("hex", 5), ("prism", 3), ("tet", 3), ("quad", 7)])
def test_matches_numpy(cuda, kind, n):
    import torch

    if kind == "tet":
        from test_gpu_fast_assembly import tets
        t, x, c = tets(n)
    else:
        t, x, c = {"hex": mesh.structured_hexes, "prism": mesh.extruded_prisms, "quad": mesh.structured_quads}[kind](n)
    b = x.shape[1] + 1
    d = NavierStokesFV1(dim=b - 1)
    d.set_mesh(t, x, c)
    rp, ci = d.pattern()
    v = (2 * mesh.uniform(3, ci.size * b * b) - 1).reshape(-1, b, b)
    u = (2 * mesh.uniform(4, x.shape[0] * b) - 1).reshape(-1, b)
    y = torch.full((u.size,), float("nan"), dtype=torch.float64, device=cuda)
    d.bsr_mv(torch.from_numpy(v.ravel()).to(cuda), torch.from_numpy(u.ravel()).to(cuda), y)
    ref, mag = np.zeros(u.shape, np.longdouble), np.zeros(u.shape)
    row = np.repeat(np.arange(x.shape[0]), np.diff(rp))
    np.add.at(ref, row, np.einsum("qij,qj->qi", v.astype(np.longdouble), u[ci].astype(np.longdouble)))
    np.add.at(mag, row, np.einsum("qij,qj->qi", np.abs(v), np.abs(u[ci])))
    err = np.abs(y.cpu().numpy().reshape(ref.shape) - ref).astype(float)
    assert np.all(err <= 4e-16 * (b * np.diff(rp).max() / 8 + 1) * mag)
