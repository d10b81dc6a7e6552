"""The calls that a simulator makes of this framework, as cases to time and compare.

A frame of an implicit simulator finds its contact pairs, lags the friction, and then repeats:
assemble the Newton system, build the preconditioner, solve, bound the step, search along it.
A differentiable one solves adjoint systems at the converged step.  Each kind below is one of
those calls on the seeded scenes of `sgipc.scenes`:

newton       computeGradientAndHessian + calculateMovingDirection (assembly, MAS, PCG)
adjoint      a batch of adjoint solves with the parameter gradients
global       the coupled system of soft bodies and affine bodies
contacts     buildCP + buildFrictionSets, the pair search and lagged friction of a frame
line_search  energy, step bounds (ground, CCD), trial step, energy there
operators    one SpMV and one MAS application, for callers with a Krylov loop of their own
"""
import dataclasses
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "stiff-gipc_b200"))

from sgipc import _native as N  # noqa: E402
from sgipc import abd, adjoint, scenes, system  # noqa: E402

CRITERIA = {"rz": N.CRIT_RZ, "true": N.CRIT_TRUE}


def listed():
    cube = dict(scene="cube", stop="rz", tol=1e-4)
    cubes = dict(scene="two_cubes", stop="rz", tol=1e-4)
    cloth = dict(scene="cloth_sphere", n=256, cells=4000)
    return [
        # the smallest system in use: a coarse collision proxy, all launches and latency
        dict(name="newton_two_cubes5_fp64", kind="newton", n=5, precision="fp64", **cubes),
        # one free soft cube, no contact yet
        dict(name="newton_cube11_mixed", kind="newton", n=11, precision="mixed", **cube),
        # the ordinary system: two stacked cubes in contact, in both main precisions
        dict(name="newton_two_cubes21_mixed", kind="newton", n=21, precision="mixed", **cubes),
        dict(name="newton_two_cubes21_fp64", kind="newton", n=21, precision="fp64", **cubes),
        # a finer mesh, beyond what one pass of the chip holds, in the reference's precision mix
        dict(name="newton_two_cubes31_ref", kind="newton", n=31, precision="ref", **cubes),
        # cloth in many layers: about a million pairs, stiff and ill conditioned
        dict(name="newton_cloth256_mixed", kind="newton", precision="mixed", stop="rz", tol=1e-4, **cloth),
        # the backward direction: gradients of four losses at once
        dict(name="adjoint_two_cubes21_mixed", kind="adjoint", n=21, nrhs=4, precision="mixed", **cubes),
        # stiff affine bodies over a soft bed, solved together
        dict(name="global_bed500_ref", kind="global", scene="bed", n=50, layers=8, boxes=500, precision="ref",
             stop="rz", tol=1e-4),
        # the pair search and friction set-up of a frame, few pairs and very many
        dict(name="contacts_two_cubes21", kind="contacts", scene="two_cubes", n=21),
        dict(name="contacts_cloth256", kind="contacts", **cloth),
        # one trial of the line search
        dict(name="line_search_two_cubes21", kind="line_search", scene="two_cubes", n=21),
        # operators alone on a small system: latency
        dict(name="operators_cube11_ref", kind="operators", scene="cube", n=11, precision="ref"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same ranges: cubes of 5 to 31 vertices an edge (two) or 5 to 33 (one),
    cloths of 32 to 256 over spheres of 300 to 4000 cells, beds of 10 to 50 cells with 20 to
    500 boxes; soft to firm, slippery to rough; every precision; the loose stop of a simulator
    or a tight one."""
    kind = rng.choice(["newton", "newton", "newton", "adjoint", "global", "contacts", "line_search", "operators"])
    case = dict(kind=kind)
    if kind == "global":
        case.update(scene="bed", n=rng.randint(10, 50), layers=rng.randint(3, 8))
        case["boxes"] = _log_int(rng, 20, max(21, case["n"] * case["n"] // 5))
    else:
        case["scene"] = rng.choice(["cube", "two_cubes", "two_cubes", "cloth_sphere"])
        if kind in ("adjoint", "contacts") and case["scene"] == "cube":
            case["scene"] = "two_cubes"
        if kind == "adjoint":  # the rolled cloth's tight solves take seconds
            case["scene"] = "two_cubes"
        if case["scene"] == "cloth_sphere":
            case.update(n=_log_int(rng, 32, 256), cells=_log_int(rng, 300, 4000))
        else:
            top = {"adjoint": 21}.get(kind, 33 if case["scene"] == "cube" else 31)
            case["n"] = _log_int(rng, 5, top)
            if case["scene"] == "two_cubes":  # meshes that do not match
                case["top"] = max(5, int(case["n"] * rng.uniform(0.8, 1.0)))
    if case["scene"] == "cloth_sphere":
        case["friction"] = round(rng.uniform(0.05, 0.5), 3)
    else:
        case["young"] = float(_log_int(rng, 3e4, 1e6))
    if kind in ("newton", "operators"):
        case["precision"] = rng.choice(["mixed", "fp64", "ref"])
    if kind == "newton" and case["scene"] == "cloth_sphere" and case["n"] < 200:
        # a small sheet's coarsest MAS domain is too ill conditioned for FP32 inverses: those
        # solves still converge, but their iterates differ by a percent from run to run
        case["precision"] = "fp64"
    if kind == "newton":
        tight = case["scene"] != "cloth_sphere" and rng.random() < 0.3
        case.update(stop="true" if tight else "rz", tol=1e-8 if tight else 1e-4)
    if kind == "adjoint":
        # the batched mixed solve is FP32 throughout, for the loose stop; tight gradients take FP64
        case.update(precision=rng.choice(["mixed", "fp64"]), nrhs=rng.randint(1, 4))
        tight = case["precision"] == "fp64"
        case.update(stop="true" if tight else "rz", tol=1e-8 if tight else 1e-4)
    if kind == "global":
        case.update(precision=rng.choice(["fp64", "ref"]), stop="rz", tol=1e-4)
    return case


# ---- scenes ------------------------------------------------------------------------------


@functools.lru_cache(maxsize=24)
def _mesh(scene, n, cells, boxes, top, young):
    """The rest shapes, which no seed changes: (scene without contacts, bodies or None)."""
    if scene == "cloth_sphere":
        return scenes.scene_cloth_on_sphere(n, cells, contacts=False), None
    if scene == "bed":
        return scenes.scene_abd_on_bed(boxes, (n, cells, n), bed_E=young, contacts=False)
    # scenes.scene_cube and scenes.scene_two_cubes, perturbation and contacts left to _scene
    gap, size = 0.5e-3, 0.1
    if scene == "cube":
        v, t = scenes.lattice_tets(n, size, (0.0, scenes.GROUND_OFFSET + 0.05, 0.0))
        bodies = [dict(verts=v, tets=t, E=young)]
    else:
        v0, t0 = scenes.lattice_tets(n, size, (0.0, scenes.GROUND_OFFSET + gap, 0.0))
        v1, t1 = scenes.lattice_tets(top, size, (0.0, scenes.GROUND_OFFSET + 2 * gap + size, 0.0))
        bodies = [dict(verts=v0, tets=t0, E=young), dict(verts=v1, tets=t1, E=10 * young)]
    return scenes.build_tet_scene("%s%d" % (scene, n), bodies, dt=0.01, dhat_abs=1e-3, density=1000.0,
                                  nu=0.4 if scene == "cube" else 0.45, mu_friction=0.0 if scene == "cube" else 0.2,
                                  seed=1, perturb=0.0), None


def _scene(case, seed):
    """The scene at one Newton iterate of the seed: the frame's start a seeded perturbation of
    the rest pose, seeded velocities, and the iterate a little way from the start."""
    sc, bodies = _mesh(case["scene"], case["n"], case.get("cells", case.get("layers", 0)), case.get("boxes", 0),
                       case.get("top", case["n"]), case.get("young", 1e5))
    rng = np.random.default_rng([seed, case["n"]])
    free = (sc.boundary_type == 0)[:, None]
    vel = np.zeros_like(sc.rest_vertexes)
    x0, body = sc.o_vertexes.copy(), sc.body_of_vertex
    noise = 1e-4
    if case["scene"] == "two_cubes":
        d = rng.normal(size=3)
        vel[body == 1] = d / np.linalg.norm(d)
    elif case["scene"] == "cloth_sphere":
        noise = 1e-6
        vel[body == 1] = (0.0, -0.5, 0.0)
        x0[body == 1] += np.array([1.0, 0.0, 1.0]) * rng.uniform(-2e-3, 2e-3, 3)
    elif case["scene"] == "bed":
        noise = 2e-5
    x0 += free * rng.uniform(-noise, noise, x0.shape)
    x = x0 + free * rng.uniform(-0.2 * noise, 0.2 * noise, x0.shape)
    xt = scenes.inertial_target(x0, vel, sc.boundary_type, sc.params["dt"])
    if bodies is not None:  # falling boxes get seeded velocities; the resting ones stay at rest
        v = np.where(bodies["resting"][:, None], 0.0, rng.normal(scale=0.1, size=(len(bodies["q"]), 3)))
        qt = bodies["q"].copy()
        qt[:, :3] += bodies["dt"] ** 2 * np.asarray(scenes.GRAVITY) + 1e-3 * bodies["dt"] * v
        bodies = dict(bodies, q_tilde=qt)
    params = dict(sc.params)
    if "friction" in case:
        params.update(frictionRate=case["friction"], gd_frictionRate=case["friction"])
    return dataclasses.replace(sc, vertexes=x, o_vertexes=x0, xTilta=xt, velocities=vel, params=params), bodies


def _pair_capacity(case):
    if case["scene"] == "cloth_sphere":
        return 30 * case["n"] ** 2 + 20000
    if case["scene"] == "bed":
        return 400 * case["boxes"] + 20000
    return 90 * case["n"] ** 2 + 2000


def prepare(case, seed):
    """The context of the scene with the frame's contacts in place, and the case's own inputs."""
    sc, bodies = _scene(case, seed)
    g = system.GIPC(sc, max_rhs=case.get("nrhs", 1), pair_capacity=_pair_capacity(case))
    s = dict(case=case, g=g)
    if case["kind"] == "global":
        s["body"] = torch.tensor(sc.body_of_vertex, dtype=torch.int32, device="cuda")
        g.buildCP(body=s["body"])
    else:
        g.buildCP()
        if sc.params["frictionRate"] > 0.0 and case["kind"] != "contacts":
            g.buildFrictionSets()
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def uniform(shape, a):
        return torch.empty(shape, dtype=torch.float64, device="cuda").uniform_(-a, a, generator=gen)

    if "precision" in case:
        s["config"] = system.PCGSolverConfig(precision=case["precision"], criterion=CRITERIA[case.get("stop", "rz")],
                                             global_tol_rate=case.get("tol", 1e-4),
                                             max_iter_ratio=1.0 if case.get("stop") == "true" else 0.3)
    if case["kind"] == "adjoint":
        s["dLdx"] = uniform((case["nrhs"], 3 * sc.nv), 1e-3)
    elif case["kind"] == "contacts":  # a frame's buffers, as large as the scene may need
        cap, ng = _pair_capacity(case), len(sc.surf_verts)
        i32, f64 = torch.int32, torch.float64
        s["frame"] = {k: torch.zeros(shape, dtype=dt, device="cuda") for k, shape, dt in (
            ("pairs", (cap, 4), i32), ("ccd_pairs", (cap, 4), i32), ("mat_index", (cap,), i32),
            ("ground_pairs", (ng,), i32), ("fric_pairs", (cap, 4), i32), ("fric_lambda", (cap,), f64),
            ("fric_coord", (cap, 2), f64), ("fric_basis", (cap, 6), f64), ("fric_gd_lambda", (ng,), f64))}
    elif case["kind"] == "line_search":
        # towards the inertial target, as a first Newton step goes, at a step that collides
        s["dir"] = (g.tet.vertexes - g.tet.xTilta + uniform((sc.nv, 3), 2e-4)).reshape(-1).contiguous()
        s["base"] = g.tet.vertexes.clone()
        s["surf"] = torch.tensor(np.asarray(sc.surf_verts, np.int32), device="cuda")
        s["ccd"] = g.buildCP(update=False)["ccd_pairs"].contiguous()
    elif case["kind"] == "operators":
        g.computeGradientAndHessian()
        s["mas"] = system.MASPreconditioner(g)
        s["mas"].setPreconditioner(case["precision"])
        s["v"] = uniform((3 * sc.nv,), 1.0)
    elif case["kind"] == "global":
        g.computeGradientAndHessian()
        part = g.contactPartition(bodies["abd_first"])
        cap = 2 * max(part["abd_blocks"][0].numel(), part["fem_blocks"][0].numel(), 1)
        sysm = abd.ABDSystem(bodies, max_abd_blocks=cap, max_fem_blocks=cap)
        s.update(bodies=bodies, cap=cap, abd=sysm, pre=abd.ABDPreconditioner(sysm), mas=system.MASPreconditioner(g),
                 gls=abd.GlobalLinearSystem(g, sysm), q=torch.tensor(bodies["q"], device="cuda"),
                 qt=torch.tensor(bodies["q_tilde"], device="cuda"))
    return s


# ---- one pass ----------------------------------------------------------------------------


def run(s):
    return RUN[s["case"]["kind"]](s)


def _newton(s):
    g = s["g"]
    g.computeGradientAndHessian()
    g.calculateMovingDirection(s["config"])
    return {"dx": g.moveDir, "rhs": g.rhs()}


def _adjoint(s):
    g, c = s["g"], s["config"]
    g.computeGradientAndHessian()
    dE, dv, lam, _ = adjoint.adjoint(g, s["dLdx"], precision=c.precision, tol=c.global_tol_rate, criterion=c.criterion)
    return {"dLdE": dE, "dLdv0": dv, "lambda": lam, "rhs": g.rhs()}


def _global(s):
    g, b, c = s["g"], s["bodies"], s["config"]
    g.computeGradientAndHessian()
    pt = g.contactPartition(b["abd_first"], s["cap"])
    s["abd"].setup_abd_system_gradient_hessian(s["q"], s["qt"], b["kappa"], b["dt"], point_grad=pt["point_grad"],
                                               abd_blocks=pt["abd_blocks"], fem_blocks=pt["fem_blocks"],
                                               fem_boundary=g.tet.BoundaryType)
    s["pre"].assemble()
    s["mas"].setPreconditioner(c.precision)
    rhs = s["gls"].right_hand_side()
    x, dx, _ = s["gls"].solve_linear_system(rhs, tol=c.global_tol_rate, criterion=c.criterion)
    nb = 12 * len(b["q"])
    return {"x": x, "points_dx": dx, "rhs_bodies": rhs[:nb], "rhs": rhs[nb:]}


def _contacts(s):
    g, t = s["g"], s["g"].tet
    out = g.buildCP()
    num = g.buildFrictionSets()
    for name, kept in s["frame"].items():
        found = out[name] if name in out else getattr(t, name)
        kept[:len(found)].copy_(found)
    return dict(s["frame"], cp_num=np.array(out["cp_num"]), cp_num_last=np.array(num), gp_num=out["gp_num"])


def _line_search(s):
    g = s["g"]
    x = g.tet.vertexes
    x.copy_(s["base"])
    e0 = g.computeEnergy()
    alpha = g.ground_largestFeasibleStepSize(0.8, s["dir"], s["surf"])
    if s["ccd"].shape[0]:
        alpha = min(alpha, g.self_largestFeasibleStepSize(0.8, s["dir"], s["ccd"]))
    g.step_forward(alpha, s["base"], s["dir"])
    return {"e0": e0, "e1": g.computeEnergy(), "alpha": alpha, "x": x}


def _operators(s):
    return {"Av": s["g"].spmv(s["v"]), "Mv": s["mas"].preconditioning(s["v"])}


RUN = dict(newton=_newton, adjoint=_adjoint, contacts=_contacts, line_search=_line_search, operators=_operators)
RUN["global"] = _global


# ---- what a pass cannot do without -------------------------------------------------------


def _sizes(case):
    """(vertices, tets, triangles, hinges, pairs) of a case's scene, pairs to a few percent."""
    n = case["n"]
    if case["scene"] == "cube":
        return n ** 3, 5 * (n - 1) ** 3, 0, 0, 0
    if case["scene"] == "two_cubes":
        m = case.get("top", n)
        return n ** 3 + m ** 3, 5 * (n - 1) ** 3 + 5 * (m - 1) ** 3, 0, 0, 49 * n * n
    if case["scene"] == "cloth_sphere":
        return n * n + 1.2 * case["cells"], 5 * case["cells"], 2 * (n - 1) ** 2, 3 * (n - 1) ** 2, 15 * n * n
    return (n + 1) ** 2 * (case["layers"] + 1) + 8 * case["boxes"], 5 * n * n * case["layers"], 0, 0, 16 * case["boxes"]


def work(case):
    """Bytes: the element, vertex and pair inputs read once, the results written once.  Flops:
    about 3000 for a tet's gradient and projected Hessian, 1500 for a pair's; for a solve, the
    SpMV (18 per stored 3x3 block, both triangles) and one 48x48 product a domain and level for
    each iteration, at the iteration counts seen."""
    v, t, f, h, p = _sizes(case)
    state = 120 * v + 120 * t + 52 * f + 152 * h
    pairs = (32 + 72) * p
    blocks = 13 * v + 10 * f / 2 + 4 * p
    domains = 1.1 * v / 16 * 1.3
    iteration = 18 * blocks + 2 * 48 * 48 * domains + 30 * v
    assembly = 3000 * t + 800 * f + 300 * h + 2 * 1500 * p
    kind = case["kind"]
    if kind == "contacts":
        surf = v if f else 6 * case["n"] ** 2 * 2
        return {"bytes": 100 * surf + (36 + 16 + 8 + 16 + 48) * p, "flops": 600 * p + 200 * surf}
    if kind == "line_search":
        return {"bytes": 2 * (state + 64 * p) + 96 * v + 112 * p, "flops": 2 * (100 * t + 60 * f + 200 * p) + 1500 * p}
    if kind == "operators":
        return {"bytes": 76 * blocks / 2 + 48 * v + 4 * 48 * 48 * domains / 2, "flops": iteration}
    its = {"cube": 2.0, "two_cubes": 1.5, "cloth_sphere": 0.9, "bed": 0.15}[case["scene"]] * case["n"]
    its *= 4.0 if case["stop"] == "true" else 1.0
    rhs = case.get("nrhs", 1)
    out = 48 * v + (rhs * 8 * (t + 6 * v) if kind == "adjoint" else 0)
    return {"bytes": state + pairs + out, "flops": assembly + rhs * its * iteration}


def tolerance(case):
    """contacts: whole numbers, and friction data computed term by term.  operators: FP32 MAS
    inverses.  line_search: sums of 64-bit terms; the CCD's step is a short iteration.  A solve
    to a true residual of 1e-8 leaves the condition number's worth of it.  A solve stopped by
    r.z <= 1e-4 r0.z0 is as exact as its last step: one iteration more or less moves dx by a
    percent or so."""
    kind = case["kind"]
    if kind == "contacts":
        return {"rel": 1e-9, "max": 1e-6}
    if kind == "operators":
        return {"rel": 1e-9 if case["precision"] == "fp64" else 1e-5, "max": 1e-3}
    if kind == "line_search":
        return {"rel": 1e-9, "max": 1e-6}
    if case["stop"] == "true":
        return {"rel": 1e-4, "max": 1e-2}
    return {"rel": 0.02, "max": 0.5}


# ---- the same in 64 bits -----------------------------------------------------------------


def _decode(pairs):
    """Kinds (0 PP, 1 PE, 2 PT, 3 EE, 4 to 6 mollified EE, PE, PP) and vertices of pair codes."""
    x, y, z, w = pairs.long().unbind(1)
    edge = x >= 0
    kind = torch.where(edge, torch.where(w >= 0, 3, 4),
                       torch.where(z < 0, torch.where(y < 0, 6, 0), torch.where(w < 0, torch.where(y < 0, 5, 1), 2)))
    v = torch.stack([torch.where(edge, x, -x - 1)] + [torch.where(u < 0, -u - 1, u) for u in (y, z, w)], 1)
    return kind, v


def _dot(a, b):
    return (a * b).sum(-1)


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=-1)


def _dist2(kind, p):
    """Squared distances of pairs of one kind, p (k, 4, 3)."""
    a, b, c, d = p.unbind(1)
    if kind in (0, 6):
        return _dot(a - b, a - b)
    if kind in (1, 5):
        n = _cross(b - a, c - a)
        return _dot(n, n) / _dot(c - b, c - b)
    n = _cross(c - b, d - b) if kind == 2 else _cross(b - a, d - c)
    s = _dot(a - b, n) if kind == 2 else _dot(c - a, n)
    return s * s / _dot(n, n)


def _pair_energy(g, x):
    t, p = g.tet, g.params
    kind, v = _decode(t.pairs)
    total = x.new_zeros(())
    for k in range(7):
        i = v[kind == k]
        if not len(i):
            continue
        i = i.clamp(max=len(x) - 1)
        ratio = _dist2(k, x[i]) / p["dHat"]
        e = p["kappa"] * p["dHat"] ** 2 * (ratio - 1) ** 2 * torch.log(ratio) ** 2
        if k >= 4:  # nearly parallel edges: the mollifier of |e0 x e1|^2
            m = i[:, {4: [0, 1, 2, 3], 5: [0, 3, 1, 2], 6: [0, 2, 1, 3]}[k]]
            q, r = x[m], t.rest_vertexes[m]
            n = _cross(q[:, 1] - q[:, 0], q[:, 3] - q[:, 2])
            ex = 1e-3 * ((r[:, 1] - r[:, 0]) ** 2).sum(1) * ((r[:, 3] - r[:, 2]) ** 2).sum(1)
            c = _dot(n, n) / ex
            e = e * (2 * c - c * c)
        total = total + e.sum()
    return total


def _friction_energy(g, x):
    t, p = g.tet, g.params
    eps = math.sqrt(p["fDhat"]) * p["dt"]
    u3, total = x - t.o_vertexes, x.new_zeros(())
    if len(t.fric_pairs):
        kind, v = _decode(t.fric_pairs)
        a, b = t.fric_coord.unbind(1)
        one, zero = torch.ones_like(a), torch.zeros_like(a)
        weight = torch.stack([torch.stack(w, 1) for w in ([one, -one, zero, zero], [one, a - 1, -a, zero],
                                                          [one, a + b - 1, -a, -b], [1 - a, a, b - 1, -b])])
        w = weight[kind.clamp(max=3), torch.arange(len(v), device=v.device)]
        rel = (w[:, :, None] * u3[v.clamp(max=len(x) - 1)]).sum(1)
        u = torch.einsum("pk,pkc->pc", rel, t.fric_basis.reshape(-1, 3, 2))
        m = torch.sqrt(_dot(u, u) + 1e-300)
        f = torch.where(m > eps, m, m * m * (eps - m / 3) / eps ** 2 + eps / 3)
        total = total + p["frictionRate"] * (t.fric_lambda * f * (kind <= 3)).sum()
    if len(t.fric_gd_pairs):
        u = u3[t.fric_gd_pairs.long()][:, [0, 2]]
        m = torch.sqrt(_dot(u, u) + 1e-300)
        f = torch.where(m > eps, m - eps / 2, m * m / (2 * eps))
        total = total + p["gd_frictionRate"] * (t.fric_gd_lambda * f).sum()
    return total


def _energy(g, x):
    """The incremental potential whose gradient is the right-hand side."""
    t, p, sc = g.tet, g.params, g.scene
    dt2 = p["dt"] ** 2
    on = lambda a: torch.as_tensor(np.asarray(a, np.int64), device=x.device)  # noqa: E731
    total = 0.5 * (t.masses[:, None] * (x - t.xTilta) ** 2).sum()
    q = x[on(sc.tets)]
    F = (q[:, 1:] - q[:, :1]).transpose(1, 2) @ t.DmInverses.reshape(-1, 3, 3)
    J = torch.linalg.det(F)
    mu, lam = t.lengthRate, t.volumeRate
    total = total + dt2 * (t.volum * 0.5 * (mu * ((F * F).sum((1, 2)) - 3) + lam * (J - 1 - mu / lam) ** 2)).sum()
    if len(sc.tris):
        q = x[on(sc.tris)]
        F = (q[:, 1:] - q[:, :1]).transpose(1, 2) @ t.triDmInverses.reshape(-1, 2, 2)
        s = torch.linalg.norm(F, dim=1) - 1
        stretch = (s * s + p["strainRate"] * s.clamp(min=0) ** 3).sum(1)
        total = total + dt2 * (t.area * (p["stretchStiff"] * stretch + p["shearStiff"] * _dot(F[:, :, 0], F[:, :, 1]) ** 2)).sum()
        both = on((np.asarray(sc.hinge_adj) >= 0).all(1).nonzero()[0])
        i = torch.cat([on(sc.hinges), on(sc.hinge_adj)], 1)[both]
        length = torch.linalg.norm(t.rest_vertexes[i[:, 0]] - t.rest_vertexes[i[:, 1]], dim=1)
        quad = torch.einsum("hij,hik,hjk->h", t.quad_bending_Q.reshape(-1, 4, 4)[both], x[i], x[i])
        total = total + dt2 * p["bendStiff"] * 0.5 * (length * quad).sum()
    if len(t.ground_pairs):
        d2 = (x[t.ground_pairs.long(), 1] - p["ground_offset"]) ** 2
        total = total - p["kappa"] * ((d2 - p["dHat"]) ** 2 * torch.log(d2 / p["dHat"])).sum()
    return total + _pair_energy(g, x) + _friction_energy(g, x)


def _gradient(g):
    x = g.tet.vertexes.clone().requires_grad_()
    _energy(g, x).backward()
    return (x.grad * (g.tet.BoundaryType == 0)[:, None]).reshape(-1)


def _tet_matrix(g):
    """Element matrices (T, 12, 12) of the tets: the second derivative of the energy density in
    F, its negative eigenvalues set to zero, in the element's corner coordinates."""
    t, sc = g.tet, g.scene
    q = g.tet.vertexes[torch.as_tensor(np.asarray(sc.tets, np.int64), device="cuda")]
    D = t.DmInverses.reshape(-1, 3, 3)
    F = (q[:, 1:] - q[:, :1]).transpose(1, 2) @ D

    def density(f, mu, lam):
        a, b, c = f.unbind(1)
        j = torch.dot(a, torch.linalg.cross(b, c))
        return 0.5 * (mu * (f * f).sum() + lam * (j - 1 - mu / lam) ** 2)

    H = torch.func.vmap(torch.func.hessian(density))(F, t.lengthRate, t.volumeRate).reshape(-1, 9, 9)
    w, V = torch.linalg.eigh(H)
    H = (V * w.clamp(min=0)[:, None]) @ V.transpose(1, 2)
    corner = torch.cat([-D.sum(1, keepdim=True), D], 1)  # dF_ij / dx_ai = corner[a, j]
    B = torch.einsum("taj,ik->tijak", corner, torch.eye(3, dtype=D.dtype, device=D.device)).reshape(-1, 9, 12)
    return (t.volum * g.params["dt"] ** 2)[:, None, None] * (B.transpose(1, 2) @ H @ B)


def _matrix_product(g):
    """v -> A v for a scene of tets without contacts, and the inverses of A's diagonal."""
    K = _tet_matrix(g)
    i = torch.as_tensor(np.asarray(g.scene.tets, np.int64), device="cuda")
    dof = (3 * i[:, :, None] + torch.arange(3, device="cuda")).reshape(-1, 12)
    m = g.tet.masses.repeat_interleave(3)

    def product(v):
        return (m * v).index_add_(0, dof.reshape(-1), torch.einsum("tij,tj->ti", K, v[dof]).reshape(-1))

    diag = m.clone().index_add_(0, dof.reshape(-1), torch.diagonal(K, dim1=1, dim2=2).reshape(-1))
    return product, 1.0 / diag


def _solve(g, b):
    product, inv = _matrix_product(g)
    x, r = torch.zeros_like(b), b.clone()
    z = inv * r
    p, rz = z.clone(), _dot(r, z)
    stop = 1e-13 * torch.linalg.norm(b)
    for k in range(6000):
        q = product(p)
        a = rz / _dot(p, q)
        x, r = x + a * p, r - a * q
        z = inv * r
        rz, old = _dot(r, z), rz
        p = z + (rz / old) * p
        if k % 50 == 49 and torch.linalg.norm(r) <= stop:
            return x
    return None


def _friction_lambda(g, x):
    t, p = g.tet, g.params
    kind, v = _decode(t.pairs)
    d2 = x.new_zeros(len(v))
    for k in range(4):
        d2[kind == k] = _dist2(k, x[v[kind == k].clamp(max=len(x) - 1)])
    d2, h = d2[kind <= 3], p["dHat"]
    log = torch.log(d2 / h)
    lam = -p["kappa"] * 2 * torch.sqrt(d2) * (2 * log * log * (d2 - h) + 2 * log * (d2 - h) ** 2 / d2)
    e2 = (x[t.ground_pairs.long(), 1] - p["ground_offset"]) ** 2
    slope = -2 * (e2 - h) * torch.log(e2 / h) - (e2 - h) ** 2 / e2
    return lam, -p["kappa"] * 2 * torch.sqrt(e2) * slope


def exact(case, seed):
    """Gradients of the energy by automatic differentiation, and the matrix of scenes without
    contacts from the density's second derivatives.  A direction that the loose stop cut short
    has no such value, nor has the order of the pairs or the advancing CCD's step."""
    s = prepare(case, seed)
    g, kind = s["g"], case["kind"]
    if kind == "newton":
        b = _gradient(g)
        dx = _solve(g, b) if case["stop"] == "true" and case["scene"] == "cube" and case["n"] <= 21 else None
        return {"dx": dx, "rhs": b}
    if kind in ("adjoint", "global"):
        return {"rhs": _gradient(g)}
    if kind == "contacts":
        found = zip(("fric_lambda", "fric_gd_lambda"), _friction_lambda(g, g.tet.o_vertexes))
        return {k: torch.cat([v, torch.zeros_like(s["frame"][k][len(v):])]) for k, v in found}
    if kind == "line_search":
        return {"e0": float(_energy(g, g.tet.vertexes))}
    return {"Av": _matrix_product(g)[0](s["v"])} if case["scene"] == "cube" else None
