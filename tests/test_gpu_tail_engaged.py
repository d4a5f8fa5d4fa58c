"""Solves in which the kernel of the lower levels runs (the report counts fewer launches than with the tuning key
"tail" 0), at the edges of its rule: 8 right-hand sides, 12 as three panels of 4, few sweeps in FP32, and a batch
without shifts, where its clusters wait for SMs beside the other branches of a graph.

Both solves stop at ||b - A u|| <= 1e-9 ||b||.  A = ⋆0⁻¹ K + I is self-adjoint for ⋆0 with eigenvalues >= 1, so
the solutions differ by at most sqrt(max ⋆0 / min ⋆0) 2e-9 ||b||, the ratio below 16 on these meshes.  The cycles
differ in last bits alone: the same number of steps."""
import numpy as np
import pytest

from conftest import uniform

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _make(dec, mesh, levels, **opts):
    if mesh == "ico":
        return dec.MultigridData(dec.meshes.icosahedron(), levels, shift=1.0, project_radius=1.0, **opts)
    coarse = dec.meshes.triangulated_grid(mesh[0] - 1, mesh[1] - 1, 1.0, 1.0, False)
    return dec.MultigridData(coarse, levels, shift=1.0, **opts)


def _rhs(mg, nrhs):
    return torch.tensor(np.stack([uniform(23 + j, mg.n) for j in range(nrhs)]), device="cuda")


def _close(got, ref, b):
    assert float((got - ref).norm(dim=1).max()) <= 8e-9 * float(b.norm(dim=1).max())


@pytest.mark.parametrize("mesh,levels", [("ico", 4), ("ico", 6), ((9, 9), 3), ((17, 13), 2)])
@pytest.mark.parametrize("nrhs,block", [(4, 0), (8, 0), (12, 4)])
@pytest.mark.parametrize("precision,pre,post,inner,mu", [(1, 0, 2, 3, 1), (0, 0, 2, 3, 1), (1, 3, 3, 1, 1), (1, 1, 1, 2, 2)])
def test_solves(dec, mesh, levels, nrhs, block, precision, pre, post, inner, mu):
    u, rep = [], []
    for on in (0, 1):
        dec.tune_clear()
        dec.tune_set("tail", on)
        mg = _make(dec, mesh, levels, precision=precision, pre=pre, post=post, inner_cycles=inner, mu=mu, rhs_block=block)
        b = _rhs(mg, nrhs)
        x, r = mg.solve(torch.zeros_like(b), b, rtol=1e-9, max_iters=60, use_initial_guess=False)
        u.append(x)
        rep.append(r)
    dec.tune_clear()
    # V(0,2) in FP32 over 81 or 221 coarsest vertices: level by level with more than 4 right-hand sides
    declines = mesh in ((9, 9), (17, 13)) and (precision, pre, post) == (1, 0, 2) and nrhs > 4
    assert (rep[1].launches == rep[0].launches) if declines else (rep[1].launches < rep[0].launches)
    assert rep[0].converged and rep[1].converged and rep[0].iterations == rep[1].iterations
    _close(u[1], u[0], b)


def test_batch_without_shifts(dec):
    groups = [("ico", 4, 8, dict(precision=1, pre=0, post=2, inner_cycles=3)), ("ico", 5, 1, dict(precision=0)),
              ((9, 9), 3, 5, dict(precision=0, pre=2, post=2)), ("ico", 6, 4, dict(precision=1)),
              ((17, 13), 2, 12, dict(precision=1, rhs_block=4)), ("ico", 6, 32, dict(precision=1, pre=0, post=2))]
    out, tot = [], []
    for on in (0, 1):
        dec.tune_clear()
        dec.tune_set("tail", on)
        mgs = [_make(dec, mesh, levels, **opts) for mesh, levels, _, opts in groups]
        bs = [_rhs(mg, g[2]) for mg, g in zip(mgs, groups)]
        batch = dec.Batch(mgs)
        for _ in range(3):   # repeated: the branches meet in other orders
            us = [torch.zeros_like(b) for b in bs]
            reps, t = batch.solve(us, bs, rtol=1e-9, max_iters=60)
        out.append(us)
        tot.append((t.launches, t.converged, [r.iterations for r in reps]))
    dec.tune_clear()
    assert tot[1][0] < tot[0][0] and tot[0][1:] == tot[1][1:] and tot[1][1] == 1
    for got, ref, b in zip(out[1], out[0], bs):
        _close(got, ref, b)
