"""The dense products of the coarsest level: row counts off the four a CTA takes, column counts around the ones
loaded together, every panel width; the inverse and the shifted solves through the eigendecomposition."""
import numpy as np
import pytest

from conftest import uniform

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("nx,ny", [(3, 3), (5, 2), (7, 5), (10, 8), (13, 13)])   # 9, 10, 35, 80, 169 vertices
@pytest.mark.parametrize("nrhs", [1, 2, 4, 7, 16, 32, 33])
@pytest.mark.parametrize("shifted", [False, True])
def test_coarsest_level_alone(dec, nx, ny, nrhs, shifted):
    """A solve on two levels above that coarsest one reaches 1e-10 in 40 steps (a wrong row would leave its
    error to the smoother, which takes hundreds), by the operator itself."""
    grid = dec.meshes.triangulated_grid(float(nx - 1), float(ny - 1), 1.0, 1.0, False)
    mg = dec.MultigridData(grid, 2, shift=0.0 if shifted else 0.05, center="barycenter", precision=0, coarse_max=170 if nx * ny > 42 else 0,
                           coarse_solver=2 if shifted else 0)
    shifts = np.linspace(0.02, 3.0, nrhs) if shifted else None
    b = torch.tensor(uniform(7, nrhs * mg.n).reshape(nrhs, mg.n), device="cuda")
    u = torch.zeros_like(b)
    _, rep = mg.solve(u, b, rtol=1e-10, max_iters=40, shifts=shifts, use_initial_guess=False)
    assert rep.converged == 1
    A = mg.level_op(0)
    for j in range(nrhs):
        r = b[j] - A.apply(u[j].clone()) - (float(shifts[j]) if shifted else 0.0) * u[j]
        assert float(r.norm()) <= 1.01e-10 * float(b[j].norm())
