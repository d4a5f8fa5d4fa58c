"""The inverse geometric ⋆1 applied on two streams in turn: the operator keeps one set of vectors, and an apply
waits for the result of the one before to be written out.  The loop's sums run in a fixed order, so a
right-hand side gives the same bits every time."""
import pytest

from conftest import uniform

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("nx,ny", [(12, 9), (340, 331)])
def test_two_streams_in_turn(dec, nx, ny):
    m = dec.meshes.triangulated_grid(nx - 1, ny - 1, 1.0, 1.0, False)
    g = dec.Mesh(m.points, m.ev0, m.ev1, m.te0, m.te1, m.te2, m.edge_orientation, m.tri_orientation)
    inv = dec.hodge_operator(1, g, inverse=True, hodge="geometric")
    xs = [torch.tensor(uniform(k, g.ne), device="cuda") for k in range(2)]
    want = [inv @ x for x in xs]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = []
    for k in range(40):
        with torch.cuda.stream(streams[k % 2]):
            got.append(inv @ xs[k % 2])
    torch.cuda.synchronize()
    for k, y in enumerate(got):
        assert torch.equal(y, want[k % 2])


def test_more_operators_than_pooled_results(dec):
    """The results that the host reads are slots of one page, 256 at a time: operators beyond them, and after
    some were given back."""
    m = dec.meshes.triangulated_grid(3.0, 2.0, 1.0, 1.0, False)
    g = dec.Mesh(m.points, m.ev0, m.ev1, m.te0, m.te1, m.te2, m.edge_orientation, m.tri_orientation)
    star = dec.hodge_operator(1, g, hodge="geometric")
    x = torch.tensor(uniform(5, g.ne), device="cuda")
    ops = []
    for k in range(300):
        ops.append(dec.hodge_operator(1, g, inverse=True, hodge="geometric"))
        y = ops[-1] @ x
        assert float((star @ y + x).norm()) <= 1e-10 * float(x.norm())
    del ops[::2]
    bad = x.clone()
    bad[0] = float("nan")
    for op in ops + [dec.hodge_operator(1, g, inverse=True, hodge="geometric") for _ in range(100)]:
        with pytest.raises(dec.DecError):
            op @ bad
        assert float((star @ (op @ x) + x).norm()) <= 1e-10 * float(x.norm())
