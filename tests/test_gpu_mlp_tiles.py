"""How the tcgen05 engine hands its 128-sample tiles to the CTAs: fewer tiles than CTAs, a partial round only,
full rounds with and without a remainder."""
import numpy as np
import pytest

from conftest import uniform

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [1, 128 * 147 + 1, 128 * 148, 128 * 148 + 1, 128 * 148 * 8 - 1, 128 * 148 * 8, 128 * 148 * 8 + 1,
                               128 * 148 * 9 + 5])
def test_eval_tiles(dec, n):
    """The engines differ in the order of their FP32 sums alone, and where that flips a BF16 rounding of a hidden
    unit: the bounds of the engines' own comparison."""
    m = dec.SmootherMLP(7)
    x = torch.tensor(uniform(3, 16 * n).reshape(n, 16), device="cuda", dtype=torch.float32)
    y1, y2 = m.eval(x, tensor_cores=1), m.eval(x, tensor_cores=2)
    d, scale = (y1 - y2).abs(), float(y1.abs().max())
    assert float(d.max()) <= 2e-3 * scale
    assert float((d <= 1e-5 * scale).float().mean()) >= 0.99 or n == 1


@pytest.mark.parametrize("level,nrhs", [(1, 1), (3, 1), (4, 32), (5, 13), (5, 32), (6, 4), (6, 32)])
def test_smoothing_tiles(dec, level, nrhs):
    """Equal right-hand sides lie in different tiles and stay equal bit for bit; the engines agree as in
    their own comparison of cycles."""
    mg = dec.MultigridData(dec.meshes.icosahedron(), level, shift=1.0, center="circumcenter", project_radius=1.0,
                           precision=1, smoother=3, pre=1, post=1)
    mlp = dec.SmootherMLP(4)
    mg.set_smoother_mlp(mlp)
    b = torch.tensor(uniform(9, mg.n), device="cuda").expand(nrhs, mg.n).contiguous()
    out = {}
    for engine in ("mma", "tcgen05"):
        mlp.set_engine(engine)
        u = mg.cycles(torch.zeros_like(b), b, 1)
        assert bool((u == u[0]).all())
        out[engine] = u[0].cpu().numpy()
    assert np.linalg.norm(out["mma"] - out["tcgen05"]) <= 1e-3 * np.linalg.norm(out["mma"])
