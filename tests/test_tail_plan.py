"""The programs planned for the kernel of the lower multigrid levels, checked on the host
(tail_plan_check.cpp): vectors that the layout reserved, and no access to another CTA's memory out of order."""
import subprocess

import pytest

from conftest import PKG_DIR, ROOT

JACOBI, CHEBYSHEV, CG = 0, 1, 2


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = tmp_path_factory.mktemp("tail") / "tail_plan_check"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{PKG_DIR / 'csrc'}", f"-I{ROOT / 'include'}",
                    str(ROOT / "tests" / "tail_plan_check.cpp"), "-o", str(exe)], check=True, timeout=300)

    def run(hierarchy, smoother, precision=0, pre=3, post=3, mu=1, inner=1, coarse_solver=0, K=1, npanels=1, cycles=1):
        line = [smoother, precision, pre, post, mu, inner, coarse_solver, len(hierarchy) - 1, K, npanels, 3, cycles,
                len(hierarchy)] + [v for level in hierarchy for v in level]
        out = subprocess.run([str(exe)], input=" ".join(map(str, line)) + "\n", capture_output=True, text=True, check=True,
                             timeout=120).stdout.splitlines()
        assert [f for f in out if f.startswith("fault")] == []
        return out[0].split()
    return run


def sphere(levels):
    """Icosphere levels, finest first: vertices, off-diagonal slots, slots of the restriction, A P present."""
    return [(10 * 4 ** k + 2, 6 if k else 5, 0 if k == 0 else 6 if k > 1 else 5, int(k > 0)) for k in range(levels, -1, -1)]


def grid(nx, ny, levels):
    nv, ne, nt = nx * ny, nx * (ny - 1) + (nx - 1) * ny + (nx - 1) * (ny - 1), 2 * (nx - 1) * (ny - 1)
    out = [(nv, 6, 0, 0)]
    for _ in range(levels):
        nv, ne, nt = nv + ne, 2 * ne + 3 * nt, 4 * nt
        out.insert(0, (nv, 6, 6, 1))
    return out


HIERARCHIES = {"sphere2": sphere(2), "sphere3": sphere(3), "sphere4": sphere(4), "sphere5": sphere(5), "sphere6": sphere(6),
               "grid3x3.5": grid(3, 3, 5), "grid5x4.4": grid(5, 4, 4), "grid9x9.3": grid(9, 9, 3), "grid17x13.2": grid(17, 13, 2)}


@pytest.mark.parametrize("mesh", HIERARCHIES)
@pytest.mark.parametrize("pre,post", [(0, 2), (1, 2), (0, 3), (3, 3), (1, 1)])
@pytest.mark.parametrize("K,npanels", [(1, 1), (4, 1), (8, 1), (4, 3)])
def test_stationary_programs(check, mesh, pre, post, K, npanels):
    on = 0
    for smoother in (JACOBI, CHEBYSHEV):
        for precision in (0, 1):
            for mu, inner, cycles in ((1, 1, 1), (1, 3, 3), (2, 2, 0), (2, 1, 2)):
                for coarse_solver in (0, 1):
                    on += check(HIERARCHIES[mesh], smoother, precision, pre, post, mu, inner, coarse_solver, K, npanels, cycles)[0] == "on"
    assert on > 0


@pytest.mark.parametrize("mesh", HIERARCHIES)
@pytest.mark.parametrize("pre,post", [(0, 2), (2, 0), (1, 2), (3, 3)])
@pytest.mark.parametrize("K,npanels", [(1, 1), (2, 1), (8, 1), (4, 3)])
def test_krylov_programs(check, mesh, pre, post, K, npanels):
    on = 0
    for mu, inner, cycles in ((1, 1, 1), (1, 3, 3), (2, 2, 0), (2, 1, 2)):
        on += check(HIERARCHIES[mesh], CG, 0, pre, post, mu, inner, 0, K, npanels, cycles)[0] == "on"
    assert on > 0


@pytest.mark.parametrize("smoother,mu", [(CHEBYSHEV, 1), (CG, 2)])
def test_long_programs_are_refused(check, smoother, mu):
    """Cycle counts are unrolled: a program is at most 65,536 phases (5 MB), whatever the count."""
    for cycles, refused in ((5, False), (50, False), (20000, True), (65535, True)):
        out = check(HIERARCHIES["sphere3"], smoother, cycles=cycles, mu=mu)
        assert out[0] == "on" and ("refused" in out) == refused and int(out[3]) <= 65536
    out = check(HIERARCHIES["sphere6"], smoother, mu=2, cycles=5)   # what dec_inverse_laplacian asks for by default
    assert out[0] == "on" and "refused" not in out
