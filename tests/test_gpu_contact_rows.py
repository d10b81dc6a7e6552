"""Rows of the contact matrix against the oracle's assembly, at the sizes where the row kernels
change: a warp or a CTA per row (128 incidences), windows of 40 columns, batches of 16 pairs a
half-warp, every pair kind (mollified ones included) and
rows of fixed vertices; and rows of thousands of columns, which are split.

The pairs are synthetic (random vertices of two small cubes, d-hat wider than the scene), so a row
can be given any length.  Tolerance: the same products in 64 bits, summed in another order; a row
of m terms differs by at most about m eps of its largest term, 1e-12 for the longest here, and
the pair geometry's own rounding grows with the pair's conditioning: 1e-9 of the largest block, the
bound of the other assembly tests.
"""
import dataclasses

import numpy as np
import pytest

import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA device", allow_module_level=True)

from sgipc import scenes, system  # noqa: E402


def _pairs(rng, nv, hub, columns, repeats, mollified):
    """Pairs that give vertex `hub` about `columns` other columns and `repeats` more incidences,
    and a background of random pairs of every kind."""
    other = np.setdiff1d(rng.permutation(nv), [hub])
    out = [(-hub - 1, w, -1, -1) for w in other[:columns]]
    near = other[:max(3, min(columns, 12))]
    for _ in range(repeats):
        a, b, c = rng.choice(near, 3, replace=False)
        out.append([(-hub - 1, a, -1, -1), (-hub - 1, a, b, -1), (-hub - 1, a, b, c), (hub, a, b, c)][rng.integers(4)])
    for _ in range(60):
        a, b, c, d = rng.choice(nv, 4, replace=False)
        kinds = [(-a - 1, b, -1, -1), (-a - 1, b, c, -1), (-a - 1, b, c, d), (a, b, c, d)]
        if mollified:
            kinds += [(a, b, c, -d - 1), (-a - 1, -b - 1, c, -d - 1), (-a - 1, -b - 1, -c - 1, -d - 1)]
        out.append(kinds[rng.integers(len(kinds))])
    return np.asarray(out, np.int32)[rng.permutation(len(out))]


@pytest.mark.parametrize("columns,repeats,mollified", [(1, 0, False), (7, 1, True), (15, 112, False), (15, 113, True),
                                                       (15, 114, False), (39, 0, False), (40, 40, True),
                                                       (41, 60, False), (81, 0, True), (330, 1000, True)])
def test_rows_match_the_oracle(columns, repeats, mollified):
    rng = np.random.default_rng(columns + repeats)
    sc = scenes.scene_two_cubes(6, seed=4)
    hub = int(rng.integers(sc.nv))
    pairs = _pairs(rng, sc.nv, hub, columns, repeats, mollified)
    fp = pairs[rng.permutation(len(pairs))[:len(pairs) // 2 + 1]]
    lam = rng.uniform(0.5, 2.0, len(fp))
    coord = rng.uniform(0.1, 0.4, (len(fp), 2))
    basis = np.linalg.qr(rng.normal(size=(len(fp), 3, 2)))[0]
    btype = sc.boundary_type.copy()
    btype[rng.choice(sc.nv, 20, replace=False)] = 1
    sc = dataclasses.replace(sc, pairs=pairs, fric_pairs=fp, fric_lambda=lam, fric_coord=coord, fric_basis=basis,
                             boundary_type=btype, params=dict(sc.params, dHat=0.2, kappa=1.0),
                             o_vertexes=sc.vertexes + rng.uniform(-1e-3, 1e-3, sc.vertexes.shape))
    g = system.GIPC(sc)
    g.computeGradientAndHessian()
    rows, cols, vals = g.export_bcoo()
    b, orow, ocol, oval, _ = oracle.assemble(sc)
    assert np.array_equal(rows, orow) and np.array_equal(cols, ocol)
    assert np.abs(vals - oval).max() <= 1e-9 * np.abs(oval).max()
    assert np.abs(g.rhs().cpu().numpy() - b).max() <= 1e-9 * np.abs(b).max()
    # the transposed lists: A times a vector against the upper blocks and their transposes
    x = rng.normal(size=3 * sc.nv)
    y = g.spmv(torch.tensor(x, device="cuda")).cpu().numpy()
    ref = oracle.spmv(orow, ocol, oval, sc.nv, x)
    assert np.abs(y - ref).max() <= 1e-9 * np.abs(ref).max()
    # the same sums on every run
    g.computeGradientAndHessian()
    assert np.array_equal(g.export_bcoo()[2], vals)
    g.close()


@pytest.mark.parametrize("copies", [1, 40])
def test_pairs_that_name_a_vertex_twice(copies):
    """Every way in which two places of a pair can hold one vertex: all of its blocks count, as in the
    oracle (friction pairs: a barrier pair of that kind is at distance zero).  40 copies of each
    give the rows of a CTA.  Tolerance as above."""
    rng = np.random.default_rng(copies)
    sc = scenes.scene_two_cubes(5, seed=4)
    shapes = [(0, 0), (0, 1), (0, 0, 1), (0, 1, 0), (1, 0, 0), (0, 1, 1), (0, 0, 0),
              (0, 0, 1, 2), (0, 1, 0, 2), (0, 1, 2, 0), (1, 0, 0, 2), (1, 0, 2, 0), (1, 2, 0, 0),
              (0, 0, 1, 1), (0, 1, 0, 1), (0, 1, 1, 0), (0, 0, 0, 1), (1, 0, 0, 0), (0, 1, 2, 3)]
    fp = []
    for _ in range(copies):
        v = rng.choice(12, 4, replace=False)
        for s in shapes:
            u = [int(v[k]) for k in s]
            fp.append([-u[0] - 1] + u[1:] + [-1] * (4 - len(u)))
            if len(u) == 4:
                fp.append(u)
    fp = np.asarray(fp, np.int32)[rng.permutation(len(fp))]
    sc = dataclasses.replace(sc, pairs=np.zeros((0, 4), np.int32), fric_pairs=fp,
                             fric_lambda=rng.uniform(0.5, 2.0, len(fp)), fric_coord=rng.uniform(0.1, 0.4, (len(fp), 2)),
                             fric_basis=np.linalg.qr(rng.normal(size=(len(fp), 3, 2)))[0],
                             o_vertexes=sc.vertexes + rng.uniform(-1e-3, 1e-3, sc.vertexes.shape))
    g = system.GIPC(sc)
    g.computeGradientAndHessian()
    rows, cols, vals = g.export_bcoo()
    b, orow, ocol, oval, _ = oracle.assemble(sc)
    assert np.array_equal(rows, orow) and np.array_equal(cols, ocol)
    assert np.abs(vals - oval).max() <= 1e-9 * np.abs(oval).max()
    assert np.abs(g.rhs().cpu().numpy() - b).max() <= 1e-9 * np.abs(b).max()
    x = rng.normal(size=3 * sc.nv)
    ref = oracle.spmv(orow, ocol, oval, sc.nv, x)
    assert np.abs(g.spmv(torch.tensor(x, device="cuda")).cpu().numpy() - ref).max() <= 1e-9 * np.abs(ref).max()
    g.close()


def test_transposed_blocks_are_exact_copies():
    """Off the diagonal A e_j read at row i equals A e_i read at row j to the last bit, for rows of warps
    and of CTAs (a product with a unit vector adds one static and one contact entry to zeros)."""
    rng = np.random.default_rng(5)
    sc = scenes.scene_two_cubes(6, seed=4)
    hub = int(rng.integers(sc.nv))
    pairs = _pairs(rng, sc.nv, hub, 60, 150, True)
    fp = pairs[rng.permutation(len(pairs))[:len(pairs) // 2]]
    sc = dataclasses.replace(sc, pairs=pairs, fric_pairs=fp, fric_lambda=rng.uniform(0.5, 2.0, len(fp)),
                             fric_coord=rng.uniform(0.1, 0.4, (len(fp), 2)),
                             fric_basis=np.linalg.qr(rng.normal(size=(len(fp), 3, 2)))[0],
                             params=dict(sc.params, dHat=0.2, kappa=1.0),
                             o_vertexes=sc.vertexes + rng.uniform(-1e-3, 1e-3, sc.vertexes.shape))
    g = system.GIPC(sc)
    g.computeGradientAndHessian()
    e = torch.eye(3 * sc.nv, dtype=torch.float64, device="cuda")
    A = torch.stack([g.spmv(e[k]) for k in range(3 * sc.nv)])
    block = torch.arange(3 * sc.nv, device="cuda") // 3
    off = block[:, None] != block
    assert torch.equal(A[off], A.T[off])
    g.close()


def _wide(rng, nv, hub, columns, fan):
    """Pairs that give `hub` about `columns` other columns: `fan` of them three or four at a time with
    the same two neighbours (a corner of a large triangle), the rest alone; and some of each twice."""
    other = np.setdiff1d(rng.permutation(nv), [hub])
    rng.shuffle(other)
    a, b = other[:2]
    far = other[2:columns]
    out = [(-w - 1, hub, a, b) for w in far[:fan]] + [(-hub - 1, w, -1, -1) for w in far[fan:]]
    out += [(-w - 1, hub, a, -1) for w in far[::7]] + [(hub, a, b, w) for w in far[::11]] + [(-a - 1, b, -1, -1)]
    return np.asarray(out, np.int32)[rng.permutation(len(out))]


@pytest.mark.parametrize("n,columns,fan,hub", [(10, 44, 20, 0.5), (10, 90, 0, 0.0), (10, 999, 600, 1.0),
                                               (18, 5000, 2500, 0.3), (18, 5830, 0, 0.0), (34, 39300, 3000, 0.0),
                                               (34, 39300, 0, 0.05)])
def test_split_rows_match_the_oracle(n, columns, fan, hub):
    """Rows of up to 39 300 columns (983 windows: more than are listed at a time), the hub's columns
    above it, below it or both; same blocks, gradient and product as the oracle's."""
    rng = np.random.default_rng(columns + fan)
    sc = scenes.scene_cube(n, seed=4)
    pairs = _wide(rng, sc.nv, int(hub * (sc.nv - 1)), columns, fan)
    btype = sc.boundary_type.copy()
    btype[rng.choice(sc.nv, 20, replace=False)] = 1
    sc = dataclasses.replace(sc, pairs=pairs, boundary_type=btype, params=dict(sc.params, dHat=0.2, kappa=1.0))
    g = system.GIPC(sc, max_rhs=1)
    g.computeGradientAndHessian()
    rows, cols, vals = g.export_bcoo()
    b, orow, ocol, oval, _ = oracle.assemble(sc)
    assert np.array_equal(rows, orow) and np.array_equal(cols, ocol)
    assert np.abs(vals - oval).max() <= 1e-9 * np.abs(oval).max()
    assert np.abs(g.rhs().cpu().numpy() - b).max() <= 1e-9 * np.abs(b).max()
    x = rng.normal(size=3 * sc.nv)
    ref = oracle.spmv(orow, ocol, oval, sc.nv, x)
    assert np.abs(g.spmv(torch.tensor(x, device="cuda")).cpu().numpy() - ref).max() <= 1e-9 * np.abs(ref).max()
    g.computeGradientAndHessian()
    assert np.array_equal(g.export_bcoo()[2], vals)
    g.close()


def test_split_rows_of_a_mesh_beyond_the_bitmap():
    """More vertices than the bitmap of a split has columns (2^18): a hub whose columns lie on both sides
    of that line, windows across it."""
    sc = scenes.scene_cloth_on_sphere(520, 300, contacts=False)
    assert sc.nv > 1 << 18
    rng = np.random.default_rng(1)
    hub = sc.nv - 3000
    w = np.sort(np.concatenate([rng.choice((1 << 18) - 1, 2000, replace=False),
                                rng.choice(np.arange(1 << 18, hub), 700, replace=False), np.arange(hub + 1, sc.nv, 2)]))
    pairs = np.stack([-hub - 1 + 0 * w, w, -1 + 0 * w, -1 + 0 * w], 1).astype(np.int32)[rng.permutation(len(w))]
    sc = dataclasses.replace(sc, pairs=pairs, ground_pairs=sc.ground_pairs[:0], params=dict(sc.params, dHat=4.0, kappa=1.0))
    assert ((sc.vertexes[w] - sc.vertexes[hub]) ** 2).sum(1).max() < 4.0
    g = system.GIPC(sc, max_rhs=1)
    g.computeGradientAndHessian()
    base = dataclasses.replace(sc, pairs=pairs[:0])
    g0 = system.GIPC(base, max_rhs=1)
    g0.computeGradientAndHessian()
    grad = (g.rhs() - g0.rhs()).cpu().numpy().reshape(-1, 3)
    e = torch.zeros(3 * sc.nv, dtype=torch.float64, device="cuda")
    X, R = sc.vertexes.reshape(-1), sc.rest_vertexes.reshape(-1)
    want = np.zeros((sc.nv, 3, 3))  # the hub's rows of the contact matrix, by column vertex
    gw = np.zeros((sc.nv, 3))
    for p in pairs:
        vid, _, gr, H = oracle.barrier_pair(p, X, R, 4.0, 1.0)
        for a, va in enumerate(vid):
            gw[va] += gr[3 * a:3 * a + 3]
        k = list(vid).index(hub)
        for a, va in enumerate(vid):
            want[va] += H[3 * k:3 * k + 3, 3 * a:3 * a + 3]
    for q in range(3):
        e.zero_()
        e[3 * hub + q] = 1.0
        col = (g.spmv(e) - g0.spmv(e)).cpu().numpy().reshape(-1, 3)  # A e: entry (vertex, p) of column (hub, q)
        assert np.abs(col - want[:, q, :]).max() <= 1e-9 * np.abs(want).max()
    free = sc.boundary_type == 0
    assert np.abs(np.abs(grad[free]) - np.abs(gw[free])).max() <= 1e-9 * np.abs(gw).max()
    g.close()
    g0.close()
