"""Vectors <-> panels: every panel width, vertex counts around a tile, and padded last panels.

From u = 0 a V-cycle is linear, so a right-hand side scaled by a power of two gives its column scaled by the
same power bit for bit, wherever the panels put it."""
import numpy as np
import pytest

from conftest import uniform

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("nrhs", [1, 2, 3, 4, 7, 8, 13, 16, 31, 32, 33, 70])
@pytest.mark.parametrize("mesh", ["31", "32", "33", "ico4"])
def test_columns_keep_their_place(dec, mesh, nrhs):
    if mesh == "ico4":   # 2,562 vertices
        mg = dec.MultigridData(dec.meshes.icosahedron(), 4, shift=1.0, center="circumcenter", project_radius=1.0, precision=0)
    else:                # one refinement of a strip of 2 x k vertices: 3 (2 k - 1) of them
        k = {"31": 5, "32": 6, "33": 43}[mesh]
        mg = dec.MultigridData(dec.meshes.triangulated_grid(float(k - 1), 1.0, 1.0, 1.0, False), 1, shift=1.0,
                               center="barycenter", precision=0)
        assert mg.n == 3 * (2 * k - 1)
    b0 = torch.tensor(uniform(3, mg.n), device="cuda")
    scale = torch.tensor([2.0 ** (j % 9 - 4) for j in range(nrhs)], device="cuda", dtype=torch.float64)
    b = scale[:, None] * b0
    u = mg.cycles(torch.zeros_like(b), b.contiguous(), 2)
    assert torch.equal(u, scale[:, None] * (u[0] / scale[0]))
    r = b0 - mg.level_op(0).apply(u[0] / scale[0])   # the column is the solution's, in the vertices' order
    assert float(r.norm()) <= 0.5 * float(b0.norm())


@pytest.mark.parametrize("n,nrhs", [(4, 3), (5, 32), (6, 9)])
def test_first_residual(dec, n, nrhs):
    """The solve's first pass over b (rows four at a time and the rest): right-hand sides that differ in scale
    by powers of two stop on the same step, at the same relative residual."""
    mg = dec.MultigridData(dec.meshes.icosahedron(), n, shift=1.0, center="circumcenter", project_radius=1.0, precision=0)
    b0 = torch.tensor(uniform(5, mg.n), device="cuda")
    scale = torch.tensor([2.0 ** (j % 9 - 4) for j in range(nrhs)], device="cuda", dtype=torch.float64)
    b = (scale[:, None] * b0).contiguous()
    u = torch.zeros_like(b)
    mg.solve(u, b, rtol=1e-9)
    assert torch.equal(u, scale[:, None] * (u[0] / scale[0]))
    A = mg.level_op(0)
    assert float((b0 - A.apply(u[0] / scale[0])).norm()) <= 1.01e-9 * float(b0.norm())
