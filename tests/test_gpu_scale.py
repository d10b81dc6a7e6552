"""Beyond shared-memory residency: a cloth 150^2 on a 12^3 cube (about 24 000 vertices,
more block rows than the persistent solve's CTAs hold in one SpMV pass, self and
cloth-cube contacts).  The persistent solve then runs without resident rows and domain
inverses, in several passes per phase.  Properties checked: every precision meets its
r.z criterion with the reported relative residual equal (1e-6) to one recomputed by the
FP64 SpMV; persistent vs graph FP64 solves within 1e-9.
"""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

from sgipc import scenes, system  # noqa: E402
from sgipc import _native as N  # noqa: E402


@pytest.fixture(scope="module")
def big():
    sc = scenes.scene_cloth_on_cube(150, 12, seed=2)
    assert sc.nv > 148 * 128   # more rows than one SpMV pass of the grid covers
    g = system.GIPC(sc)
    g.computeGradientAndHessian()
    yield sc, g
    g.close()


@pytest.mark.parametrize("prec", ["fp64", "mixed", "ref"])
def test_large_scene_solve_meets_criterion(big, prec):
    sc, g = big
    system.MASPreconditioner(g).setPreconditioner(prec)
    b = g.rhs()
    x, st = system.PCGSolver(g, system.PCGSolverConfig(precision=prec)).solve(b)
    assert st.status == N.OK and st.iterations > 0
    assert abs(st.rz) <= 1e-4 * st.rz0 * (1 + 1e-9)
    res = float((b - g.spmv(x)).norm() / b.norm())
    assert st.rel_residual == pytest.approx(res, rel=1e-6)


def test_large_scene_persistent_and_graph_agree(big, monkeypatch):
    sc, g = big
    system.MASPreconditioner(g).setPreconditioner("fp64")
    solver = system.PCGSolver(g, system.PCGSolverConfig(precision="fp64"))
    xa, sa = solver.solve(g.rhs())
    monkeypatch.setenv("SGIPC_PCG_GRAPH", "1")
    xb, sb = solver.solve(g.rhs())
    monkeypatch.delenv("SGIPC_PCG_GRAPH")
    assert abs(sa.iterations - sb.iterations) <= 1
    if sa.iterations == sb.iterations:
        assert float((xa - xb).abs().max() / xb.abs().max()) < 1e-9


@pytest.mark.parametrize("n", [28, 33])
def test_banks_by_cta_and_by_half_cta_agree_with_graph(n, monkeypatch):
    """The position pass with fewer level-1 banks than CTAs (28^3) and with more (33^3, two banks a
    CTA at a time, the last CTA one): the graph of kernels, which sums in another order, reaches the
    same solution.  Both stop at a true residual of 1e-10 |b|, so each is within 1e-10 cond(A) |x| of
    the exact one, and cond(A) is below 1e4 here (the mass term)."""
    sc = scenes.scene_cube(n, touching=True)
    g = system.GIPC(sc)
    g.computeGradientAndHessian()
    mas = system.MASPreconditioner(g)
    mas.setPreconditioner("fp64")
    banks = (int(mas.info()[1][1]) + 15) // 16
    assert sc.nv > 148 * 128 and (banks > 148) == (n == 33)
    b = torch.randn(3 * sc.nv, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(n))
    solver = system.PCGSolver(g, system.PCGSolverConfig(precision="fp64", criterion=N.CRIT_TRUE, global_tol_rate=1e-10,
                                                        max_iter_ratio=1.0))
    xa, sa = solver.solve(b)
    monkeypatch.setenv("SGIPC_PCG_GRAPH", "1")
    xb, sb = solver.solve(b)
    monkeypatch.delenv("SGIPC_PCG_GRAPH")
    assert sa.status == N.OK and sb.status == N.OK
    for x in (xa, xb):
        assert float((b - g.spmv(x)).norm() / b.norm()) < 1.1e-10
    assert float((xa - xb).norm() / xb.norm()) < 1e-6
    g.close()
