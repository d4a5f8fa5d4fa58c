"""Full multigrid with the stationary smoothers in the kernel of the lower levels, against the per-level kernels
(tuning key "tail" 0).  Full multigrid prolongs an iterate into every level before it cycles, so V(0,2) ends in
the correction form there.  Every row, transfer and sum keeps its arithmetic except the dense coarsest product
(FP64, summed in another order): 1e-12 of scale, as for the cycles."""
import numpy as np
import pytest

from conftest import uniform

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("mesh,levels", [("ico", 3), ("ico", 4), ("ico", 5), ("ico", 6), ((9, 9), 3), ((5, 4), 4), ((17, 13), 3)])
@pytest.mark.parametrize("nrhs", [1, 5])
@pytest.mark.parametrize("pre,post,mu", [(0, 2, 1), (0, 2, 2), (1, 2, 1), (0, 3, 1)])
def test_full_multigrid(dec, mesh, levels, nrhs, pre, post, mu):
    if mesh == "ico":
        coarse, radius = dec.meshes.icosahedron(), 1.0
    else:
        coarse, radius = dec.meshes.triangulated_grid(mesh[0] - 1, mesh[1] - 1, 1.0, 1.0, False), 0.0
    out, launches = [], []
    for on in (0, 1):
        dec.tune_clear()
        dec.tune_set("tail", on)
        mg = dec.MultigridData(coarse, levels, shift=1.0, project_radius=radius, smoother=1, pre=pre, post=post, mu=mu,
                               precision=0)
        b = torch.tensor(np.stack([uniform(11 + j, mg.n) for j in range(nrhs)]), device="cuda")
        out.append([dec.full_multigrid(b, mg, c).cpu().numpy() for c in (1, 3, 0)])
        launches.append(mg.solve(torch.zeros_like(b), b, rtol=1e-6, max_iters=60, use_initial_guess=False)[1].launches)
    dec.tune_clear()
    assert launches[1] < launches[0]   # the kernel of the lower levels did run
    for ref, got in zip(*out):
        assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()
