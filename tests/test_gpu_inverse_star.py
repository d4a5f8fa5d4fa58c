"""The inverse geometric ⋆1 (a BiCGSTAB loop on the device) at the sizes where its kernels change shape:
fewer rows than a block, whole blocks and a remainder, more rows than the grid (grid-stride), FP32, the
alpha / beta epilogue, a zero and a non-finite right-hand side.  ⋆1 applied to the result gives -x back: the
solve stops at 1e-14 of the right-hand side and refuses above 1e-10."""
import numpy as np
import pytest

from conftest import uniform

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _mesh(dec, nx, ny):
    m = dec.meshes.triangulated_grid(nx - 1, ny - 1, 1.0, 1.0, False)
    return dec.Mesh(m.points, m.ev0, m.ev1, m.te0, m.te1, m.te2, m.edge_orientation, m.tri_orientation)


@pytest.mark.parametrize("nx,ny", [(2, 2), (5, 4), (10, 10), (33, 31), (340, 331)])
@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_inverse_undoes_the_star(dec, nx, ny, dtype):
    g = _mesh(dec, nx, ny)
    inv = dec.hodge_operator(1, g, inverse=True, hodge="geometric", dtype=dtype)
    star = dec.hodge_operator(1, g, hodge="geometric")
    tol = 1e-10 if dtype == "float64" else 1e-5   # FP32: the input and the result are rounded
    for seed in (1, 2):   # the second call reuses the vectors of the first
        x = torch.tensor(uniform(seed, g.ne), device="cuda", dtype=getattr(torch, dtype))
        back = -(star @ (inv @ x).double())
        assert float((back - x.double()).norm()) <= tol * float(x.double().norm())
    y = torch.ones_like(x)
    out = inv.apply(x, y.clone(), alpha=2.0, beta=3.0)
    assert float((out - (2.0 * (inv @ x) + 3.0)).abs().max()) <= 1e-6 * float(out.abs().max())


def test_zero_and_non_finite(dec):
    g = _mesh(dec, 12, 9)
    inv = dec.hodge_operator(1, g, inverse=True, hodge="geometric")
    z = torch.zeros(g.ne, dtype=torch.float64, device="cuda")
    assert bool((inv @ z == 0).all())
    bad = z.clone()
    bad[3] = float("nan")
    with pytest.raises(dec.DecError):
        inv @ bad
    x = torch.tensor(uniform(4, g.ne), device="cuda")
    star = dec.hodge_operator(1, g, hodge="geometric")
    assert float((star @ (inv @ x) + x).norm()) <= 1e-10 * float(x.norm())   # usable after the refusal
