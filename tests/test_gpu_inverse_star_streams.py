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
