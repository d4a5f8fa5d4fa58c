"""The lower levels of a cycle as one kernel (k_tail) against the per-level kernels it stands for (tuning
key "tail" 0): the same bits, since every row, transfer and sum keeps the per-level kernels' arithmetic
and order.  The dense coarsest product alone sums in another order, in FP64: its last bits may differ,
which the cycles above contract (1e-12 of scale for FP64 results; FP32 cycles round it away or carry one
FP32 rounding, 1e-9 after the FP64 refinement).  Sizes: one CTA (every level small), levels split over
the cluster with and without a remainder, coarse meshes whose rows are not six wide, 1 to 15 right-hand
sides, hierarchies whose finest level is outside."""
import numpy as np
import pytest

from conftest import uniform

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _coarse(dec, mesh):
    if mesh == "ico":
        return dec.meshes.icosahedron(), 1.0
    nx, ny = mesh
    return dec.meshes.triangulated_grid(nx - 1, ny - 1, 1.0, 1.0, False), 0.0


def _both(dec, make, run):
    out = []
    for on in (0, 1):
        dec.tune_clear()
        dec.tune_set("tail", on)
        out.append([t.cpu().numpy() for t in run(make())])
    dec.tune_clear()
    return out


CG = [("ico", 1, 1, 1, 3), ("ico", 4, 1, 1, 3), ("ico", 5, 3, 2, 2), ("ico", 6, 1, 1, 1), ("ico", 3, 8, 1, 4),
      ((9, 11), 2, 1, 2, 4), ((5, 5), 5, 1, 2, 3), ((3, 4), 4, 2, 1, 2), ((17, 13), 3, 7, 1, 3)]


@pytest.mark.parametrize("mesh,levels,nrhs,mu,steps", CG)
def test_krylov_cycles_same_bits(dec, mesh, levels, nrhs, mu, steps):
    coarse, radius = _coarse(dec, mesh)

    def make():
        return dec.MultigridData(coarse, levels, shift=1.0, project_radius=radius, smoother=2, pre=steps, post=steps, mu=mu)

    def run(mg):
        b = torch.tensor(np.stack([uniform(7 + j, mg.n) for j in range(nrhs)]), device="cuda")
        u = torch.tensor(np.stack([uniform(70 + j, mg.n) for j in range(nrhs)]), device="cuda")
        return mg.cycles(u.clone(), b, 2), mg.cycles(torch.zeros_like(b), b, 1), dec.full_multigrid(b, mg, 2)

    for ref, got in zip(*_both(dec, make, run)):
        np.testing.assert_array_equal(got, ref)


@pytest.mark.parametrize("mesh,levels", [((9, 9), 3), ((3, 4), 5)])
def test_singular_operator_same_bits(dec, mesh, levels):
    """The Laplacian itself (shift 0) with W-cycles: a Krylov smoother on its coarse levels magnifies a
    single last bit."""
    coarse, _ = _coarse(dec, mesh)
    b = None

    def run(inv):
        b = inv.md.level_op(0) @ torch.tensor(uniform(3, inv.md.n), device="cuda")
        return (inv(b),)

    ref, got = _both(dec, lambda: dec.dec_inverse_laplacian(0, coarse, levels, steps=2, cycles=3), run)
    np.testing.assert_array_equal(got[0], ref[0])


CHEB = [("ico", 2, 1, 1, 3, 3, 1, 1), ("ico", 4, 2, 0, 3, 3, 1, 1), ("ico", 5, 1, 1, 0, 2, 3, 1), ("ico", 6, 1, 0, 0, 2, 3, 1),
        ("ico", 5, 15, 1, 2, 2, 2, 2), ("ico", 6, 4, 1, 1, 2, 1, 2), ((6, 5), 4, 2, 1, 0, 2, 3, 1), ((9, 6), 5, 1, 0, 2, 3, 1, 1),
        ((5, 4), 1, 3, 1, 0, 1, 1, 1)]


@pytest.mark.parametrize("smoother", [0, 1])
@pytest.mark.parametrize("mesh,levels,nrhs,precision,pre,post,inner,mu", CHEB)
def test_stationary_cycles(dec, smoother, mesh, levels, nrhs, precision, pre, post, inner, mu):
    coarse, radius = _coarse(dec, mesh)

    def make():
        return dec.MultigridData(coarse, levels, shift=1.0, project_radius=radius, smoother=smoother, pre=pre, post=post,
                                 precision=precision, inner_cycles=inner, mu=mu)

    def run(mg):
        b = torch.tensor(np.stack([uniform(7 + j, mg.n) for j in range(nrhs)]), device="cuda")
        u = torch.tensor(np.stack([uniform(70 + j, mg.n) for j in range(nrhs)]), device="cuda")
        x0, r0 = mg.solve(torch.zeros_like(b), b, rtol=1e-9, max_iters=60, use_initial_guess=False)
        x1, r1 = mg.solve(u.clone(), b, rtol=1e-9, max_iters=60)
        its = torch.tensor([r0.iterations, r1.iterations, r0.converged, r1.converged])
        return x0, x1, mg.cycles(u.clone(), b, 2), its

    ref, got = _both(dec, make, run)
    for k, tol in ((0, 1e-9 if precision else 1e-12), (1, 1e-9 if precision else 1e-12), (2, 1e-12)):
        assert np.abs(got[k] - ref[k]).max() <= tol * np.abs(ref[k]).max()
    np.testing.assert_array_equal(got[3], ref[3])


def test_coarsest_smoothed_and_level_steps(dec):
    """The smoother on the coarsest level (its products in the per-level order: the same bits), sweep counts
    changed after a solve, and a hierarchy solved directly at a middle level."""
    ico = dec.meshes.icosahedron()
    b = None

    def run(mg):
        b = torch.tensor(uniform(5, mg.n), device="cuda")
        out = [mg.cycles(torch.zeros_like(b), b, 2).clone()]
        mg.set_level_steps([1, 2, 3, 2, 1])
        out.append(mg.cycles(torch.zeros_like(b), b, 2))
        return out

    for opts in (dict(coarse_solver=1), dict(coarse_solver=1, smoother=0, mu=2)):
        ref, got = _both(dec, lambda: dec.MultigridData(ico, 4, shift=1.0, project_radius=1.0, **opts), run)
        for r, g in zip(ref, got):
            np.testing.assert_array_equal(g, r)
    ref, got = _both(dec, lambda: dec.MultigridData(ico, 4, shift=1.0, project_radius=1.0, coarse_max=170), run)
    for r, g in zip(ref, got):
        assert np.abs(g - r).max() <= 1e-12 * np.abs(r).max()
