"""The tree far field (EB_FAR_TREE, the default engine of larger meshes).

Against the CPU oracle on sampled rows and against the symmetric kernels on
every row. FP64 is held to 1e-12 (the bar of the FP64 engines), mixed to 1e-6.
The sizes put the last cell at 1 and 31 triangles, split the bisection
unevenly and lie just above the smallest size that takes the tree; the shapes
are closed, open, in two distant parts, thin, graded, and in units far from
one (every expansion coefficient is scaled by its cluster's radius).
"""
import numpy as np
import pytest

from conftest import rel_l2
from easybem_b200 import meshes

pytestmark = pytest.mark.gpu

FP64_TOL, MIXED_TOL = 1e-12, 1e-6


def _cut(v, f, ne):
    """The first ne triangles (an open surface)."""
    return v, f[:ne]


def _two(n_u):
    v, f = meshes.torus(n_u, 0.3)
    return np.vstack([v, 0.4 * v + np.array([7.0, -3.0, 1.0])]), np.vstack([f, f + len(v)])


def _graded(level):
    v, f = meshes.icosphere(level)
    return v * np.array([3.0, 0.6, 0.15]) * (0.05 + np.exp(-2.0 * (1 + v[:, :1]))), f


MESHES = {
    "torus206": lambda: meshes.torus(206, 0.25),            # 21,012 triangles: last cell of 20
    "cut12801": lambda: _cut(*meshes.torus(206, 0.25), 12801),  # last cell of 1
    "cut12831": lambda: _cut(*meshes.torus(206, 0.25), 12831),  # last cell of 31
    "cut16416": lambda: _cut(*meshes.perturbed_icosphere(5, seed=3), 16416),
    "two": lambda: _two(165),
    "graded": lambda: _graded(5),
}


def _vectors(nodes, elems, seed):
    rng = np.random.default_rng(seed)
    return rng.normal(size=len(elems)), rng.normal(size=len(nodes))


@pytest.mark.parametrize("name", list(MESHES))
def test_tree_matches_oracle_and_symmetric_kernels(gpu_lib, oracle, name):
    oracle.set_order(4)
    nodes, elems = MESHES[name]()
    t, u = _vectors(nodes, elems, len(name))
    rows = np.sort(np.random.default_rng(1).choice(len(elems), 48, replace=False)).astype(np.int32)
    vo, qo = oracle.apply_rows(nodes, elems, t, u, rows)
    with gpu_lib.Mesh(nodes, elems) as m:
        assert m.far_engine("mixed") == "tree" and m.far_engine("fp64") == "tree"
        for prec, tol in (("fp64", FP64_TOL), ("mixed", MIXED_TOL)):
            m.set_far_engine("tree")
            v, q = m.apply_sl_dl(t, u, precision=prec)
            assert rel_l2(v[rows], vo) < tol and rel_l2(q[rows], qo) < tol
            v2, q2 = m.apply_sl_dl(t, u, precision=prec)
            assert np.array_equal(v, v2) and np.array_equal(q, q2)
            vs = m.apply_sl(t, precision=prec)
            assert rel_l2(vs[rows], vo) < tol
            d = m.apply_hypersingular(u, precision=prec)
            qs = m.apply_dl(u, precision=prec)
            assert rel_l2(qs[rows], qo) < tol
            w = m.apply_sl_p1(u, precision=prec)
            m.set_far_engine("cuda")
            assert rel_l2(w, m.apply_sl_p1(u, precision=prec)) < tol
            m.set_far_engine("sym_all")
            vd, qd = m.apply_sl_dl(t, u, precision=prec)
            assert rel_l2(v, vd) < tol and rel_l2(q, qd) < tol
            assert rel_l2(d, m.apply_hypersingular(u, precision=prec)) < 10 * tol  # differences of V's columns


@pytest.mark.parametrize("name", ["cut12801", "two"])
@pytest.mark.parametrize("nrhs", [1, 3, 5])
def test_tree_right_hand_sides(gpu_lib, name, nrhs):
    """b = 1/2 M g + K g: one column, a padded group of four, four and one."""
    nodes, elems = MESHES[name]()
    g = np.random.default_rng(nrhs).normal(size=(nrhs, len(nodes)))
    with gpu_lib.Mesh(nodes, elems) as m:
        for prec, tol in (("fp64", FP64_TOL), ("mixed", MIXED_TOL)):
            m.set_far_engine("tree")
            b = m.dirichlet_rhs(g, prec)
            m.set_far_engine("cuda")
            c = m.dirichlet_rhs(g, prec)
            for k in range(nrhs):
                assert rel_l2(b[k], c[k]) < tol


@pytest.mark.parametrize("unit", [1e-9, 1e6])
def test_tree_in_other_units(gpu_lib, unit):
    nodes, elems = meshes.torus(180, 0.3)
    t, u = _vectors(nodes, elems, 5)
    with gpu_lib.Mesh(nodes, elems) as a, gpu_lib.Mesh(nodes * unit, elems) as b:
        assert b.far_engine("fp64") == "tree"
        # the FP32 point sums have an absolute floor of 1e-12 in distance: at
        # 1e-9 they are no reference
        for prec, tol in (("fp64", FP64_TOL), ("mixed", MIXED_TOL))[:1 if unit < 1e-6 else 2]:
            v, q = a.apply_sl_dl(t, u, precision=prec)
            w, r = b.apply_sl_dl(t, u, precision=prec)
            assert rel_l2(w / unit ** 3, v) < tol and rel_l2(r / unit ** 2, q) < tol


def test_meshes_without_separated_clusters_keep_the_direct_sum(gpu_lib):
    """A tube of long strips: every cell spans it, nearly all cells are close."""
    n = 8200
    a = 2 * np.pi * np.arange(n) / n
    ring = np.stack([np.cos(a), np.sin(a), np.zeros(n)], 1)
    nodes = np.vstack([ring - [0, 0, 20.0], ring + [0, 0, 20.0]])
    i, j = np.arange(n), (np.arange(n) + 1) % n
    elems = (np.vstack([np.stack([i, j, n + j], 1), np.stack([i, n + j, n + i], 1)]) + 1).astype(np.int32)
    t, u = _vectors(nodes, elems, 9)
    with gpu_lib.Mesh(nodes, elems) as m:
        for prec, engine in (("mixed", "sym"), ("fp64", "cuda")):
            m.set_far_engine("tree")
            assert m.far_engine(prec) == engine
            v, q = m.apply_sl_dl(t, u, precision=prec)
            m.set_far_engine(engine)
            w, r = m.apply_sl_dl(t, u, precision=prec)
            assert np.array_equal(v, w) and np.array_equal(q, r)


def test_tree_follows_plan_changes(gpu_lib):
    nodes, elems = meshes.torus(170, 0.3)
    t, u = _vectors(nodes, elems, 6)
    with gpu_lib.Mesh(nodes, elems) as m:
        v, q = m.apply_sl_dl(t, u)
        m.set_plan(64)  # releases the records that the tree's descriptors point to
        w, r = m.apply_sl_dl(t, u)
        assert np.array_equal(v, w) and np.array_equal(q, r)


@pytest.mark.parametrize("ne", [1, 31, 32, 33, 127, 864, 865, 1280, 3199, 3201, 4000])
def test_small_meshes_sum_all_cell_pairs(gpu_lib, oracle, ne):
    """Cells that all lie close: one cell, whole and ragged last cells, both
    sides of the smallest tree."""
    oracle.set_order(4)
    nodes, elems = meshes.torus(100, 0.3)
    nodes, elems = _cut(nodes, elems, ne)
    t, u = _vectors(nodes, elems, ne)
    rows = np.sort(np.random.default_rng(1).choice(ne, min(ne, 64), replace=False)).astype(np.int32)
    vo, qo = oracle.apply_rows(nodes, elems, t, u, rows)
    g = np.stack([u, u[::-1], 2 * u])
    with gpu_lib.Mesh(nodes, elems) as m:
        if ne < 3200:
            assert m.far_engine("mixed") == "sym" and m.far_engine("fp64") == "sym"
        for prec, tol in (("fp64", FP64_TOL), ("mixed", MIXED_TOL)):
            m.set_far_engine("tree")
            v, q = m.apply_sl_dl(t, u, precision=prec)
            vs, qs, b, d = m.apply_sl(t, prec), m.apply_dl(u, prec), m.dirichlet_rhs(g, prec), m.apply_hypersingular(u, prec)
            p = m.apply_sl_p1(u, prec)
            assert rel_l2(v[rows], vo) < tol and rel_l2(vs[rows], vo) < tol
            m.set_far_engine("cuda")
            w, r = m.apply_sl_dl(t, u, precision=prec)
            c, e = m.dirichlet_rhs(g, prec), m.apply_hypersingular(u, prec)
            assert rel_l2(p, m.apply_sl_p1(u, prec)) < tol
            if ne == 1:  # no pair but the triangle with itself: K u = 0
                assert not q.any() and not qs.any() and not r.any()
            else:
                assert rel_l2(q[rows], qo) < tol and rel_l2(qs[rows], qo) < tol
                assert rel_l2(d, e) < 10 * tol
            assert rel_l2(b, c) < tol


@pytest.mark.parametrize("npts", [2000, 5000, 5017, 20000])
@pytest.mark.parametrize("name", ["torus206", "graded", "two"])
def test_tree_potentials(gpu_lib, oracle, name, npts):
    """Points far away, in the volume and close to the surface, several of them
    the same; ragged last groups. One point that is not finite leaves the
    others alone."""
    oracle.set_order(4)
    nodes, elems = MESHES[name]()
    t, u = _vectors(nodes, elems, npts)
    rng = np.random.default_rng(npts)
    c = nodes.mean(axis=0)
    size = np.linalg.norm(nodes - c, axis=1).max()
    pts = c + size * rng.uniform(-1.5, 1.5, size=(npts, 3))
    k = rng.integers(0, len(elems), size=npts // 4)
    tri = nodes[elems[k] - 1]
    nrm = np.cross(tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0])
    h = np.sqrt(np.linalg.norm(nrm, axis=1, keepdims=True))
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    pts[: npts // 4] = tri.mean(axis=1) + nrm * h * rng.uniform(0.5, 3.0, size=(npts // 4, 1))
    pts[-40:] = pts[-41]
    with gpu_lib.Mesh(nodes, elems) as m:
        for prec, tol in (("fp64", FP64_TOL), ("mixed", MIXED_TOL)):
            m.set_far_engine("tree")
            p = m.evaluate(pts, t, u, prec)
            assert np.array_equal(p, m.evaluate(pts, t, u, prec))
            bad = pts.copy()
            bad[5] = np.nan
            pb = m.evaluate(bad, t, u, prec)
            assert np.isnan(pb[5]) and rel_l2(np.delete(pb, 5), np.delete(p, 5)) < tol
            m.set_far_engine("cuda")
            assert rel_l2(p, m.evaluate(pts, t, u, prec)) < tol
        rows = np.linspace(0, npts - 1, 64).astype(int)
        m.set_far_engine("tree")
        assert rel_l2(m.evaluate(pts, t, u)[rows], oracle.evaluate(nodes, elems, pts[rows], t, u)) < FP64_TOL


@pytest.mark.parametrize("order", [6, 7, 9, 10, 18])
@pytest.mark.parametrize("ne", [4160, 4737, 12831])
def test_larger_rules(gpu_lib, order, ne):
    """Rules of 13 to 73 points: against the direct kernels, every row."""
    nodes, elems = _cut(*meshes.torus(206, 0.25), ne)
    t, u = _vectors(nodes, elems, order)
    with gpu_lib.Mesh(nodes, elems, order=order) as m:
        for prec, tol in (("fp64", FP64_TOL), ("mixed", MIXED_TOL)):
            m.set_far_engine("tree")
            got = [*m.apply_sl_dl(t, u, precision=prec), m.apply_sl(t, prec), m.apply_dl(u, prec)]
            m.set_far_engine("cuda")
            ref = [*m.apply_sl_dl(t, u, precision=prec), m.apply_sl(t, prec), m.apply_dl(u, prec)]
            for g, r in zip(got, ref):
                assert rel_l2(g, r) < tol


@pytest.mark.parametrize("order", [7, 9])
def test_batch_of_larger_rules(gpu_lib, order):
    """Meshes with and without separated clusters in one batch, against each alone."""
    meshes_in = [_cut(*meshes.torus(206, 0.25), ne) for ne in (12831, 640, 4737)]
    vecs = [_vectors(*x, k) for k, x in enumerate(meshes_in)]
    ms = [gpu_lib.Mesh(*x, order=order) for x in meshes_in]
    for prec, tol in (("fp64", FP64_TOL), ("mixed", MIXED_TOL)):
        bt = gpu_lib.Batch(ms, precision=prec, sl_dl=True)
        vs, qs = bt.apply_sl_dl([t for t, _ in vecs], [u for _, u in vecs])
        bt.close()
        for m, (t, u), v, q in zip(ms, vecs, vs, qs):
            w, r = m.apply_sl_dl(t, u, precision=prec)
            assert rel_l2(v, w) < tol and rel_l2(q, r) < tol
    for m in ms:
        m.close()
