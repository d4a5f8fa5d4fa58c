"""The FP64 ∧02 kernel of two triangles a thread: one triangle, odd counts, more than a block, batches, and
forms off the 16-byte boundary, which take the one-triangle kernel."""
import numpy as np
import pytest

from conftest import uniform

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def fan(dec, n):
    """n triangles around a vertex: (host mesh, device mesh)."""
    b = dec.meshes._Builder()
    for k in range(n):
        b.glue(0, k + 1, k + 2)
    ang = np.linspace(0.0, 6.0, n + 1)
    pts = np.concatenate([np.zeros((1, 3)), np.stack([np.cos(ang), np.sin(ang), 0 * ang], 1)])
    m = b.mesh(pts, None)
    return m, dec.Mesh(m.points, m.ev0, m.ev1, m.te0, m.te1, m.te2, m.edge_orientation, m.tri_orientation, center="barycenter")


def shifted(x):
    """The same values 8 bytes past a 16-byte boundary."""
    buf = torch.empty(x.numel() + 1, dtype=x.dtype, device=x.device)
    buf[1:] = x
    assert buf[1:].data_ptr() % 16 == 8
    return buf[1:]


@pytest.mark.parametrize("nt", [1, 2, 3, 511, 512, 513, 1025])
@pytest.mark.parametrize("swap", [False, True])
def test_w02_pairs(O, dec, nt, swap):
    m, g = fan(dec, nt)
    assert g.nt == nt
    w = dec.dec_wedge_product(2, 0, g) if swap else dec.dec_wedge_product(0, 2, g)
    call = (lambda f, a: w(a, f)) if swap else w
    f, a = torch.tensor(uniform(1, g.nv), device="cuda"), torch.tensor(uniform(2, g.nt), device="cuda")
    got = call(f, a).cpu().numpy()
    np.testing.assert_array_equal(call(f, shifted(a)).cpu().numpy(), got)
    om = O.mesh_from_arrays(m.points, m.ev0, m.ev1, m.te0, m.te1, m.te2, m.edge_orientation, np.zeros(nt, np.int8))
    O.orient(om)
    d = O.dualize(om, O.BARYCENTER)
    want = O.wedge(d, 2, f.cpu().numpy(), a.cpu().numpy())
    np.testing.assert_allclose(got, want, rtol=0, atol=1e-13)


@pytest.mark.parametrize("nt", [3, 514])
def test_w02_pairs_batched(dec, nt):
    """An even count keeps the vector kernel for every pair of a batch, an odd one does not."""
    _, g = fan(dec, nt)
    w = dec.dec_wedge_product(0, 2, g)
    f = torch.tensor(uniform(3, 3 * g.nv).reshape(3, g.nv), device="cuda")
    a = torch.tensor(uniform(4, 3 * g.nt).reshape(3, g.nt), device="cuda")
    got = w.batched(f, a, torch.empty_like(a))
    for k in range(3):
        assert torch.equal(got[k], w(f[k].clone(), a[k].clone()))


@pytest.mark.parametrize("level", [7, 8])   # below and above two rows for each of the chip's threads
def test_float32_rows_default(dec, level):
    """The untuned FP32 apply has the bits of one row per thread, also with alpha, beta."""
    dec.tune_clear()
    m = dec.meshes.icosphere(level)
    g = dec.Mesh(m.points, m.ev0, m.ev1, m.te0, m.te1, m.te2, m.edge_orientation, m.tri_orientation, center="circumcenter")
    L = dec.laplace_beltrami(g, "float32")
    x = torch.tensor(uniform(5, g.nv), device="cuda", dtype=torch.float32)
    y = torch.tensor(uniform(6, g.nv), device="cuda", dtype=torch.float32)
    got = L.apply(x), L.apply(x, y=y.clone(), alpha=0.5, beta=2.0)
    dec.tune_set(f"ell/f32/W7/n{int(np.log2(g.nv))}", 1)
    try:
        want = L.apply(x), L.apply(x, y=y.clone(), alpha=0.5, beta=2.0)
    finally:
        dec.tune_clear()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
