"""The calls of a frame on a side stream, with long work pending on the default stream.

Every entry point orders its work on the stream it is given; torch's side streams do not wait for
the default stream, so a memset or copy left there would land in the middle of a call, or after
it.  A fresh context runs on a side stream while the default stream multiplies matrices, and gives
what another fresh context gave on the idle default stream.

The pair search is exact and in a fixed order.  The right-hand sides differ by the order of atomic
additions (ground contacts, a body's points: FP64 rounding, 1e-12), and so do the MAS domains.  A
solve carries that on: the coupled one takes 153 to 158 iterations from run to run on an idle default
stream too, its dx moving by 1e-7.  So every solve here stops at a true residual of 1e-10 |b|, and dx
is held to 1e-6, the bound of the coupled solve's other tests.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

from sgipc import abd, scenes, system  # noqa: E402
from sgipc import _native as N  # noqa: E402

CONFIG = system.PCGSolverConfig(precision="fp64", criterion=N.CRIT_TRUE, global_tol_rate=1e-10, max_iter_ratio=1.0)


def _fem():
    sc = scenes.scene_two_cubes(7, seed=3)
    g = system.GIPC(sc, pair_capacity=4 * len(sc.pairs))
    d = torch.tensor(1e-3 * np.random.default_rng(0).standard_normal(3 * sc.nv), device="cuda")
    surf = torch.tensor(np.asarray(sc.surf_verts, np.int32), device="cuda")
    x0 = g.tet.vertexes.clone()
    g.buildCP()  # (first calls and grown buffers wait for the device)
    g.buildFrictionSets()

    def frame():
        out = g.buildCP()
        num = g.buildFrictionSets()
        g.computeGradientAndHessian()
        st = g.calculateMovingDirection(CONFIG)
        r = {"pairs": out["pairs"], "rhs": g.rhs(), "dx": g.moveDir, "energy": g.computeEnergy()}
        X, sb = system.PCGSolver(g, CONFIG).solve_batched(g.rhs().repeat(4, 1))
        a = min(g.ground_largestFeasibleStepSize(0.8, d, surf), g.self_largestFeasibleStepSize(0.8, d, out["ccd_pairs"]))
        g.step_forward(a, x0, d)
        assert st.status == N.OK and all(s.status == N.OK for s in sb)
        r.update(X=X, alpha=a, x=g.tet.vertexes, num=num)
        return r

    return frame, g.close


def _coupled():
    sc, bodies = scenes.scene_abd_on_bed(12, (6, 2, 6), seed=1, resting=0.7)
    g = system.GIPC(sc)
    sysm = abd.ABDSystem(bodies, max_abd_blocks=4000, max_fem_blocks=4000)
    pre, gls, mas = abd.ABDPreconditioner(sysm), abd.GlobalLinearSystem(g, sysm), system.MASPreconditioner(g)
    q, qt = (torch.tensor(bodies[k], device="cuda") for k in ("q", "q_tilde"))

    def frame():
        g.computeGradientAndHessian()
        pt = g.contactPartition(bodies["abd_first"])
        sysm.setup_abd_system_gradient_hessian(q, qt, bodies["kappa"], bodies["dt"], point_grad=pt["point_grad"],
                                               abd_blocks=pt["abd_blocks"], fem_blocks=pt["fem_blocks"],
                                               fem_boundary=g.tet.BoundaryType)
        pre.assemble()
        mas.setPreconditioner("fp64")
        rhs = gls.right_hand_side()
        x, dx, st = gls.solve_linear_system(rhs, tol=1e-10, criterion=N.CRIT_TRUE)  # the context's first: its buffers grow here
        assert st.status == N.OK
        return {"rhs": rhs, "dx": x, "points_dx": dx}

    def close():
        sysm.close()
        g.close()

    return frame, close


@pytest.mark.parametrize("make", [_fem, _coupled])
def test_frame_on_a_side_stream_beside_a_busy_default_stream(make):
    frame, close = make()  # the default stream's, which also loads every kernel
    ref = {k: v.clone() if torch.is_tensor(v) else v for k, v in frame().items()}
    close()
    frame, close = make()
    a = torch.randn(8192, 8192, device="cuda")
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(60):  # about a second of ordinary work, a few milliseconds of frame
        a = a @ a * 1e-2
    ahead = torch.cuda.Event()
    ahead.record()
    with torch.cuda.stream(side):
        got = frame()
        side.synchronize()
    assert not ahead.query(), "the default stream ran dry: the frame was not beside its work"
    assert got.get("num") == ref.get("num")
    for k, tol in (("pairs", 0.0), ("rhs", 1e-12), ("dx", 1e-6), ("X", 1e-6), ("points_dx", 1e-6), ("x", 1e-6)):
        if k in ref:
            d = (got[k] - ref[k]).abs().max()
            assert float(d) <= tol * float(ref[k].abs().max()), k
    for k in ("energy", "alpha"):
        assert got.get(k) == pytest.approx(ref.get(k), rel=1e-9) if k in ref else True
    torch.cuda.synchronize()
    close()
