"""A full_multigrid that the caller captured in a CUDA graph of its own: the graph keeps the sweep counts of the
capture and stays replayable after calls that drop the hierarchy's own graphs."""
import pytest

from conftest import uniform

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("opts", [dict(smoother=2, pre=3, post=3), dict(smoother=1, pre=2, post=2), dict(smoother=1, pre=0, post=2)])
@pytest.mark.parametrize("levels", [3, 6])
def test_captured_full_multigrid_outlives_the_sweep_counts(dec, opts, levels):
    mg = dec.MultigridData(dec.meshes.icosahedron(), levels, shift=1.0, project_radius=1.0, precision=0, **opts)
    b = torch.tensor(uniform(3, mg.n), device="cuda")
    want = dec.full_multigrid(b, mg, 2)
    graph, out = torch.cuda.CUDAGraph(), []
    with torch.cuda.graph(graph):
        out.append(dec.full_multigrid(b, mg, 2))
    for k in (1, 4):   # neither is the count of the capture
        mg.set_level_steps([k] * (levels + 1))
        other = dec.full_multigrid(b, mg, 2)
        # what was freed is handed out again
        junk = [dec.MultigridData(dec.meshes.icosahedron(), levels, shift=2.0, project_radius=1.0, precision=0, **opts) for _ in range(2)]
        for m in junk:
            dec.full_multigrid(b, m, 2)
        out[0].zero_()
        graph.replay()
        assert torch.equal(out[0], want) and not torch.equal(out[0], other)
