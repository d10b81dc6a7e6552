"""The forms of the persistent solve at the sizes where one takes over from another.

Up to 2048 rows the fused solve runs on one cluster of 16 CTAs with 16, 32, 64 or 128 rows each,
beyond that (and under a caller's wait limit) on a CTA per SM; FP64 vectors with four right-hand
sides take the cluster up to 256 rows and the four-phase iteration beyond.  Row counts at each of
these lines and one past it, the last CTAs with few rows or none; the grid that stamped a profiled
solve tells the form.

Every form is the same recurrence or the plain one with sums in another order, whose rounding grows
over the iterations (the longest box here moves x by 3e-3 in FP32 at a loose stop), so x itself is not
compared: every form has to reach the same true residual, |b - A x| <= tol |b| with the product taken
apart from the solve (twice that where the vectors are FP32 throughout: their own residual is a
recurrence), with r0.z0 equal to 1e-12 and the iterations within a tenth.
"""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

from sgipc import _native as N  # noqa: E402
from sgipc import scenes, system  # noqa: E402

# vertices -> lattice boxes that have them
SIZES = {128: [(4, 4, 8)], 256: [(4, 8, 8)], 257: [(3, 3, 3), (2, 5, 23)], 512: [(8, 8, 8)], 513: [(3, 3, 3), (6, 9, 9)],
         1024: [(8, 8, 16)], 1025: [(5, 5, 5), (9, 10, 10)], 1331: [(11, 11, 11)], 2047: [(3, 3, 7), (8, 8, 31)],
         2048: [(8, 16, 16)], 2049: [(9, 9, 9), (10, 11, 12)]}


@pytest.fixture(scope="module", params=sorted(SIZES))
def system_of(request):
    h, x0, bodies = 0.01, 0.0, []
    for box in SIZES[request.param]:
        v, t = scenes.box_lattice_tets(box, h, (x0, scenes.GROUND_OFFSET + 0.0005, 0.0))
        bodies.append(dict(verts=v, tets=t, E=1e5))
        x0 += box[0] * h
    sc = scenes.build_tet_scene("boxes", bodies, dt=0.01, dhat_abs=1e-3, density=1000.0, nu=0.4, mu_friction=0.0,
                                seed=1, perturb=1e-4)
    assert sc.nv == request.param
    g = system.GIPC(sc)
    g.computeGradientAndHessian()
    yield sc, g
    g.close()


@pytest.mark.parametrize("rhs", [1, 4])
@pytest.mark.parametrize("prec", ["fp64", "ref", "mixed"])
def test_forms_agree(system_of, prec, rhs, monkeypatch):
    sc, g = system_of
    mas = system.MASPreconditioner(g)
    mas.setPreconditioner(prec)
    assert mas.info()[0] >= 3  # (two levels are not fused)
    b = torch.randn(rhs, 3 * sc.nv, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(2))
    tol = {"fp64": 1e-10, "ref": 1e-10, "mixed": 1e-8 if rhs == 1 else 1e-4}[prec]
    solver = system.PCGSolver(g, system.PCGSolverConfig(precision=prec, criterion=N.CRIT_TRUE, global_tol_rate=tol,
                                                        max_iter_ratio=1.0))

    def solve():
        if rhs == 1:
            x, st = solver.solve(b[0])
            return x[None], [st]
        return solver.solve_batched(b)

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if prec != "ref":  # the form, from the CTAs of a profiled solve of the same kind
        name = ("pcg64" if prec == "fp64" else "pcg32") + ("x4" if rhs == 4 else "")
        stamps, phases = g.profile_pcg(name)
        cluster = sc.nv <= (256 if name == "pcg64x4" else 2048)
        assert (stamps.shape[0] == 16) == cluster
        assert ("fused_spmv" in phases) == (cluster or name != "pcg64x4")
        assert cluster or stamps.shape[0] >= sms
    x, st = solve()
    N.check(N.lib().sgipc_set_wait_limit(g.ctx, 1 << 40), g.ctx)  # never reached: the grid form
    if prec != "ref":
        assert g.profile_pcg(name)[0].shape[0] >= sms
    xg, sg = solve()
    N.check(N.lib().sgipc_set_wait_limit(g.ctx, 0), g.ctx)
    monkeypatch.setenv("SGIPC_PCG_FUSED", "0")
    xp, sp = solve()
    monkeypatch.delenv("SGIPC_PCG_FUSED")
    reach = tol * (2.0 if prec == "mixed" and rhs == 4 else 1.1)
    for y, sy in ((x, st), (xg, sg), (xp, sp)):
        for r in range(rhs):
            assert sy[r].status == N.OK
            assert float((b[r] - g.spmv(y[r])).norm() / b[r].norm()) <= reach
            assert abs(sy[r].iterations - st[r].iterations) <= 1 + st[r].iterations // 10
            assert abs(sy[r].rz0 - st[r].rz0) <= 1e-12 * abs(st[r].rz0)
