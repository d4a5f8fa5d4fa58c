"""The training kernels where their forms change: batches that are not multiples of 4, of the 32 samples a
slice stages or of the 256 of a chunk (the 4-byte and 16-byte copies), and feature rows of 7 slots and of
other widths."""
import numpy as np
import pytest

from conftest import uniform

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [1, 3, 31, 32, 33, 255, 256, 260, 1021, 4096, 70001])
def test_gradient_against_torch(dec, n):
    """Σ dy ∂MLP/∂params with the library's roundings (weights, features and the first hidden layer in BF16):
    1e-3 of the gradient's norm, the training kernels' stated bound (dz enters as two BF16 parts)."""
    mlp = dec.SmootherMLP(11)
    p = torch.tensor(mlp.params, device="cuda").double().requires_grad_()
    x = torch.tensor(uniform(1, 16 * n).reshape(n, 16), device="cuda", dtype=torch.float32)
    dy = torch.tensor(uniform(2, n), device="cuda", dtype=torch.float32)

    def bf(t):   # the rounded value, the gradient passed through
        return t + (t.float().bfloat16().double() - t).detach()

    w1, b1, w2, b2, w3 = p[:1024].view(64, 16), p[1024:1088], p[1088:5184].view(64, 64), p[5184:5248], p[5248:5312]
    h1 = bf(torch.relu(bf(x.double()) @ bf(w1).t() + b1))
    y = torch.relu(h1 @ bf(w2).t() + b2) @ w3 + p[5312]
    (y * dy.double()).sum().backward()
    got = mlp.grad(x, dy).double()
    assert float((got - p.grad).norm()) <= 1e-3 * float(p.grad.norm())


@pytest.mark.parametrize("level", [0, 1, 3])
def test_features(dec, level):
    """Rows of 6 slots (the icosahedron) and of 7: the features as the operator's rows give them, in FP32."""
    m = dec.meshes.icosphere(level)
    g = dec.Mesh(m.points, m.ev0, m.ev1, m.te0, m.te1, m.te2, m.edge_orientation, m.tri_orientation, center="circumcenter")
    op = dec.helmholtz(g, 1.0)
    r = torch.tensor(np.stack([uniform(5 + s, g.nv) for s in range(2)]), device="cuda")
    f, sc = dec.SmootherMLP.features(op, r)
    rp, ci, v, _ = op.csr()
    want, scale = np.zeros((2, g.nv, 16), np.float32), np.zeros((2, g.nv), np.float32)
    rh = r.cpu().numpy()
    for s in range(2):
        for i in range(g.nv):
            c, a = ci[rp[i]:rp[i + 1]], v[rp[i]:rp[i + 1]]
            d = np.float32(a[c == i].sum())
            nb, cp = rh[s][c[c != i]].astype(np.float32), a[c != i].astype(np.float32)
            big = np.float32(max(abs(np.float32(rh[s][i])), np.abs(nb).max()))
            inv = np.float32(1) / big
            want[s, i, 0] = np.float32(rh[s][i]) * inv
            want[s, i, 1:1 + len(nb)] = nb * inv
            want[s, i, 7:7 + len(nb)] = cp / d
            want[s, i, 13] = np.float32(1) - np.float32(sum(np.abs(cp), np.float32(0))) / d
            want[s, i, 14] = len(nb) / 6
            scale[s, i] = big / d
    np.testing.assert_allclose(f.cpu().numpy().reshape(2, g.nv, 16), want, rtol=0, atol=3e-6)
    np.testing.assert_allclose(sc.cpu().numpy().reshape(2, g.nv), scale, rtol=1e-6)
