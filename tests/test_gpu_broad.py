"""The GPU contact-pair search (``sgipc_build_cp``) and lagged friction set-up
(``sgipc_friction_setup``) through the C ABI.

* Against the reference's own pair checks and friction set-up, host-compiled from a reference
  checkout (``tests/golden/ref_golden.npz``, on the two scenes stored beside it): the same
  multiset of (pair, CCD candidate) rows, every pair size's MatIndex ranks 0 .. count - 1
  once, the same counters _cpNum[5] and ground pairs; the friction arrays pair for pair.
* Against the host generator (``sgipc.contacts``, itself pinned to the same goldens on the
  CPU) at the bench's size (two 21^3 cubes), on a cloth over a cube and on a rolled cloth over
  a sphere.
* Deterministic: two calls give the same arrays in the same order; the order is point-triangle
  pairs by surface point, then edge-edge pairs by edge.
* The Newton system assembled from the GPU's pairs and friction sets equals the oracle's
  assembly of the same inputs (1e-9).

Integer outputs are compared exactly; the friction forces 1e-12 relative, coordinates and
bases 1e-12 absolute (the same formulas; log and sqrt may round differently by an ulp).
"""
import os

import numpy as np
import pytest

import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

from sgipc import contacts, scenes, system  # noqa: E402

HERE = os.path.dirname(os.path.abspath(__file__))
G = np.load(os.path.join(HERE, "golden", "ref_golden.npz"))
FILES = {"cubes": "scene_two_cubes4.npz", "cloth": "scene_cloth6_cube4.npz"}


def _rows_sorted(*arrays):
    return np.array(sorted(map(tuple, np.concatenate([np.asarray(a).reshape(len(a), -1) for a in arrays], 1))))


def _sizes(p):
    return np.where(p[:, 0] >= 0, 4, np.where(p[:, 2] < 0, 2, np.where(p[:, 3] < 0, 3, 4)))


def _check_mat_index(p, mi, cp):
    """MatIndex = rank in output order among the pairs of the same size."""
    size = _sizes(p)
    for g, nv in ((2, 2), (3, 3), (4, 4)):
        assert np.array_equal(mi[size == nv], np.arange(cp[g])), nv
    assert cp[0] == len(p) and cp[1] == 0


@pytest.fixture(scope="module", params=["cubes", "cloth"])
def golden(request):
    sc = scenes.Scene.load(os.path.join(HERE, "golden", FILES[request.param]))
    g = system.GIPC(sc, pair_capacity=4096)
    yield request.param, sc, g
    g.close()


@pytest.mark.parametrize("variant", ["self", "bodies"])
def test_pairs_match_reference(golden, variant):
    tag, sc, g = golden
    q = "%s_cp_%s_" % (tag, variant)
    body = torch.tensor(G[q + "body"], device="cuda")
    out = g.buildCP(body=body, update=False)
    p, c, mi = out["pairs"].cpu().numpy(), out["ccd_pairs"].cpu().numpy(), out["mat_index"].cpu().numpy()
    assert np.array_equal(_rows_sorted(p, c), _rows_sorted(G[q + "pairs"], G[q + "ccd"]))
    assert list(out["cp_num"]) == list(G[q + "cpnum"])
    _check_mat_index(p, mi, out["cp_num"])
    assert np.array_equal(out["cp_num_dev"].cpu().numpy(), G[q + "cpnum"].astype(np.int32))
    gp = out["ground_pairs"].cpu().numpy()
    assert np.array_equal(np.sort(gp), np.sort(G[tag + "_cp_ground"])) and out["gp_num"] == len(gp)


def test_friction_sets_match_reference(golden):
    tag, sc, g = golden
    tet = system.DeviceTetraData(sc)
    cp = g.buildFrictionSets(tet)
    assert np.array_equal(tet.fric_pairs.cpu().numpy(), sc.fric_pairs)
    assert list(cp) == list(G[tag + "_lag_cpnum"])
    lam = tet.fric_lambda.cpu().numpy()
    assert np.abs(lam - sc.fric_lambda).max() <= 1e-12 * np.abs(sc.fric_lambda).max()
    assert np.abs(tet.fric_coord.cpu().numpy() - sc.fric_coord).max() <= 1e-12
    assert np.abs(tet.fric_basis.cpu().numpy().reshape(-1, 3, 2) - sc.fric_basis).max() <= 1e-12
    assert np.array_equal(tet.fric_gd_pairs.cpu().numpy(), sc.fric_gd_pairs)
    gl = tet.fric_gd_lambda.cpu().numpy()
    assert np.abs(gl - sc.fric_gd_lambda).max() <= 1e-12 * np.abs(sc.fric_gd_lambda).max()


@pytest.fixture(scope="module", params=["two_cubes21", "cloth24_cube6", "cloth_roll64_sphere"])
def large(request):
    if request.param == "two_cubes21":
        sc = scenes.scene_two_cubes(21, seed=1)
    elif request.param == "cloth24_cube6":
        sc = scenes.scene_cloth_on_cube(24, 6, seed=2)
    else:  # rolled cloth layers 0.4 mm apart: dense self-contact, about 50 000 pairs
        sc = scenes.scene_cloth_on_sphere(64, 500)
    g = system.GIPC(sc, pair_capacity=max(4 * len(sc.pairs), 4096))
    yield request.param, sc, g
    g.close()


def test_pairs_match_host_generator_and_repeat(large):
    name, sc, g = large
    pairs, ccd = contacts.find_pairs(sc.vertexes, sc.rest_vertexes, sc.surf_tris, sc.surf_edges, sc.surf_verts,
                                     sc.params["dHat"], sc.body_of_vertex, with_ccd=True)
    out = g.buildCP(update=False)
    p, c, mi = out["pairs"].cpu().numpy(), out["ccd_pairs"].cpu().numpy(), out["mat_index"].cpu().numpy()
    assert len(p) == len(pairs) > 0
    assert np.array_equal(_rows_sorted(p, c), _rows_sorted(pairs, ccd))
    _check_mat_index(p, mi, out["cp_num"])
    # the documented order: point-triangle pairs by surface point (their CCD candidates start
    # with -point - 1), then edge-edge pairs by (edge, other edge)
    pt = c[:, 0] < 0
    npt = int(pt.sum())
    assert pt[:npt].all() and not pt[npt:].any()
    pos = {int(v): i for i, v in enumerate(sc.surf_verts)}
    order = np.array([pos[-int(v) - 1] for v in c[:npt, 0]])
    assert (np.diff(order) >= 0).all()
    gp = contacts.ground_pairs(sc.vertexes, sc.surf_verts, sc.params["dHat"], sc.params["ground_offset"])
    assert np.array_equal(out["ground_pairs"].cpu().numpy(), gp)
    again = g.buildCP(update=False)
    for k in ("pairs", "ccd_pairs", "mat_index", "ground_pairs"):
        assert torch.equal(again[k], out[k]), k


def test_friction_sets_match_host_generator(large):
    name, sc, g = large
    tet = system.DeviceTetraData(sc)
    g.buildFrictionSets(tet)
    lp, lam, coord, basis, gpairs, glam = contacts.lag_friction(sc.o_vertexes, sc.pairs, sc.ground_pairs,
                                                                sc.params["dHat"], sc.params["kappa"],
                                                                sc.params["ground_offset"])
    assert np.array_equal(tet.fric_pairs.cpu().numpy(), lp)
    assert np.abs(tet.fric_lambda.cpu().numpy() - lam).max() <= 1e-12 * np.abs(lam).max()
    assert np.abs(tet.fric_coord.cpu().numpy() - coord).max() <= 1e-10
    assert np.abs(tet.fric_basis.cpu().numpy().reshape(-1, 3, 2) - basis).max() <= 1e-12
    assert np.array_equal(tet.fric_gd_pairs.cpu().numpy(), gpairs)


def test_newton_system_from_gpu_contacts_matches_oracle():
    """One Newton system whose contacts come from the GPU: the pair search at x, the friction
    sets at the start-of-step positions, then the assembly; against the oracle given the
    same pairs and friction arrays."""
    sc = scenes.scene_two_cubes(7, seed=5)
    g = system.GIPC(sc, pair_capacity=4 * len(sc.pairs))
    try:
        g.buildCP()
        g.buildFrictionSets()
        g.computeGradientAndHessian()
        rows, cols, vals = g.export_bcoo()
        b = g.rhs().cpu().numpy()
        s2 = scenes.Scene(**{**sc.__dict__})
        t = g.tet
        s2.pairs, s2.ground_pairs = t.pairs.cpu().numpy(), t.ground_pairs.cpu().numpy()
        s2.fric_pairs, s2.fric_lambda = t.fric_pairs.cpu().numpy(), t.fric_lambda.cpu().numpy()
        s2.fric_coord, s2.fric_basis = t.fric_coord.cpu().numpy(), t.fric_basis.cpu().numpy().reshape(-1, 3, 2)
        s2.fric_gd_pairs, s2.fric_gd_lambda = t.fric_gd_pairs.cpu().numpy(), t.fric_gd_lambda.cpu().numpy()
        ob, orow, ocol, oval, _ = oracle.assemble(s2)
        assert np.array_equal(rows, orow) and np.array_equal(cols, ocol)
        assert np.abs(vals - oval).max() < 1e-9 * np.abs(oval).max()
        assert np.abs(b - ob).max() < 1e-9 * np.abs(ob).max()
        assert len(s2.pairs) == len(sc.pairs)
    finally:
        g.close()


def test_capacity_is_reported():
    sc = scenes.scene_two_cubes(7, seed=5)
    g = system.GIPC(sc)
    try:
        from sgipc import _native as N

        with pytest.raises(N.SgipcError) as e:
            g.buildCP(capacity=8, update=False)
        assert e.value.status == N.CAPACITY
        assert b"capacity" in N.lib().sgipc_last_error(g.ctx)
        out = g.buildCP(update=False)  # the context stays usable
        assert out["cp_num"][0] == len(sc.pairs)
    finally:
        g.close()


def _soup_scene(kind, n, seed):
    """Loose triangles (``n`` of them, each a body of its own): ``mixed`` scatters sizes over a
    factor of 200, ``stack`` piles equal ones 0.3 d-hat apart, ``flat`` puts all in one plane."""
    rng = np.random.default_rng(seed)
    dhat = 1e-3
    size = 10.0 ** rng.uniform(-3, -0.7, n) if kind == "mixed" else np.full(n, 5e-3)
    centre = rng.uniform(0.0, 0.02, (n, 3))
    if kind == "stack":
        centre = np.stack([rng.uniform(0, 5e-3, n), 0.3 * dhat * np.arange(n), rng.uniform(0, 5e-3, n)], 1)
    tri = centre[:, None] + size[:, None, None] * rng.uniform(-1.0, 1.0, (n, 3, 3))
    if kind != "mixed":
        tri[:, :, 1] = centre[:, None, 1] if kind == "stack" else 0.01
    verts = tri.reshape(-1, 3) + np.array([0.0, scenes.GROUND_OFFSET, 0.0])
    bodies = [dict(verts=v.reshape(3, 3), tris=np.array([[0, 1, 2]]), affine=True) for v in verts.reshape(n, 9)]
    # (a soft tetrahedron far away: a scene has at least one element)
    v, t = scenes.lattice_tets(2, 0.01, (0.5, scenes.GROUND_OFFSET + 0.5, 0.5))
    return scenes.build_tet_scene("soup", [dict(verts=v, tets=t, E=1e5)] + bodies, dt=0.01, dhat_abs=dhat,
                                  density=1000.0, nu=0.4, mu_friction=0.0, seed=seed, perturb=0.0)


@pytest.mark.parametrize("kind,n", [("mixed", 1), ("mixed", 10), ("mixed", 32), ("mixed", 33), ("mixed", 341),
                                    ("mixed", 400), ("stack", 64), ("stack", 350), ("flat", 40)])
def test_pairs_of_loose_triangles(kind, n):
    """Remainders of the 32-wide groups and 1024-wide nodes, primitives of very different size,
    coincident Morton codes: the same pairs and order as the host generator finds."""
    sc = _soup_scene(kind, n, seed=n)
    pairs, ccd = contacts.find_pairs(sc.vertexes, sc.rest_vertexes, sc.surf_tris, sc.surf_edges, sc.surf_verts,
                                     sc.params["dHat"], sc.body_of_vertex, with_ccd=True)
    g = system.GIPC(sc, pair_capacity=len(pairs) + 1)
    out = g.buildCP(update=False)
    p, c = out["pairs"].cpu().numpy(), out["ccd_pairs"].cpu().numpy()
    assert len(p) == len(pairs)
    if len(p):
        assert np.array_equal(_rows_sorted(p, c), _rows_sorted(pairs, ccd))
    _check_mat_index(p, out["mat_index"].cpu().numpy(), out["cp_num"])
    ground = contacts.ground_pairs(sc.vertexes, sc.surf_verts, sc.params["dHat"], sc.params["ground_offset"])
    assert np.array_equal(out["ground_pairs"].cpu().numpy(), ground)
    if len(p) > 1:  # one place short: the counts come back, nothing is written
        with pytest.raises(Exception, match="capacity"):
            g.buildCP(update=False, capacity=len(p) - 1)
    g.close()


@pytest.mark.parametrize("points,tris,edges", [(0, 1, 1), (1, 0, 1), (1, 1, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (0, 0, 0)])
def test_surfaces_with_empty_lists(points, tris, edges):
    """Each list of the surface empty or not: the pairs that the rest gives, as the host generator finds
    them; without surface points the scene has no bounds, which is an input error (not a launch of
    no CTAs) and leaves the context usable."""
    from sgipc import _native as N

    sc = scenes.scene_two_cubes(7, seed=5)
    few = scenes.Scene(**{**sc.__dict__})
    if not points:
        few.surf_verts = sc.surf_verts[:0]
    if not tris:
        few.surf_tris = sc.surf_tris[:0]
    if not edges:
        few.surf_edges = sc.surf_edges[:0]
    g = system.GIPC(sc, pair_capacity=4 * len(sc.pairs))
    g.scene = few
    if points:
        out = g.buildCP(update=False)
        pairs, ccd = contacts.find_pairs(few.vertexes, few.rest_vertexes, few.surf_tris, few.surf_edges, few.surf_verts,
                                         few.params["dHat"], few.body_of_vertex, with_ccd=True)
        assert len(out["pairs"]) == len(pairs) and (len(pairs) > 0) == bool(tris or edges)
        if len(pairs):
            assert np.array_equal(_rows_sorted(out["pairs"].cpu().numpy(), out["ccd_pairs"].cpu().numpy()),
                                  _rows_sorted(pairs, ccd))
        ground = contacts.ground_pairs(few.vertexes, few.surf_verts, few.params["dHat"], few.params["ground_offset"])
        assert np.array_equal(out["ground_pairs"].cpu().numpy(), ground)
    else:
        with pytest.raises(N.SgipcError) as e:
            g.buildCP(update=False)
        assert e.value.status == N.BAD_INPUT
    g.scene, g._surf = sc, None
    assert g.buildCP(update=False)["cp_num"][0] == len(sc.pairs)
    g.close()


@pytest.mark.parametrize("which", ["edges", "points"])
def test_more_group_pairs_than_the_list_holds(which):
    """The search lists 64 meeting pairs of groups per query group and 1024 more, and searches what finds no
    room on the spot.  Here nearly every two groups meet: segments (or triangles) that run from one
    octant into the opposite one, 150 groups of edges (11 325 pairs for 10 624 places), or 32 groups of
    points against 110 of triangles (3520 for 3072)."""
    rng = np.random.default_rng(3)
    n = 2400  # vertices in each octant
    a, b = rng.uniform(0.01, 0.03, (n, 3)), rng.uniform(-0.03, -0.01, (n, 3))
    tris = np.stack([rng.integers(n, size=3520), n + rng.integers(n, size=3520), n + rng.integers(n, size=3520)], 1)
    tris = tris[tris[:, 1] != tris[:, 2]]
    v, t = scenes.lattice_tets(2, 0.01, (0.5, scenes.GROUND_OFFSET + 0.5, 0.5))
    verts = np.concatenate([a, b]) + np.array([0.0, scenes.GROUND_OFFSET + 0.1, 0.0])
    sc = scenes.build_tet_scene("crossing", [dict(verts=v, tets=t, E=1e5), dict(verts=verts, tris=tris, affine=True)],
                                dt=0.01, dhat_abs=1e-5, density=1000.0, nu=0.4, mu_friction=0.0, seed=1, perturb=0.0)
    few = scenes.Scene(**{**sc.__dict__})
    first = len(v)
    if which == "edges":
        few.surf_tris, few.surf_verts = sc.surf_tris[:0], first + np.arange(32)
        e = np.unique(np.stack([rng.integers(n, size=4900), n + rng.integers(n, size=4900)], 1), axis=0)[:4800]
        few.surf_edges = first + rng.permutation(e)
    else:
        few.surf_tris, few.surf_edges = first + tris, sc.surf_edges[:0]
        few.surf_verts = first + rng.permutation(2 * n)[:1024]
    pairs, ccd = contacts.find_pairs(few.vertexes, few.rest_vertexes, few.surf_tris, few.surf_edges, few.surf_verts,
                                     few.params["dHat"], few.body_of_vertex, with_ccd=True)
    assert len(pairs) > 100
    g = system.GIPC(sc, pair_capacity=len(pairs))
    g.scene = few
    out = g.buildCP(update=False)
    assert np.array_equal(_rows_sorted(out["pairs"].cpu().numpy(), out["ccd_pairs"].cpu().numpy()),
                          _rows_sorted(pairs, ccd))
    again = g.buildCP(update=False)
    assert torch.equal(again["pairs"], out["pairs"]) and torch.equal(again["mat_index"], out["mat_index"])
    g.close()
