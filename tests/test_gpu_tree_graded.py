"""The tree far field where cells of very different size meet.

A coarse cell cannot be split, so beside a finely meshed part its radius, not
the sum of the two radii, decides how fast the expansions converge. The errors
are taken on the rows of the smallest triangles alone (a norm over all rows
hides them), against the ordered-pair kernels in FP64: 1e-12 for FP64, or three
times what the symmetric FP64 kernels differ by on the same rows (rounding of
nearly cancelling double layers), and 1e-6 for mixed.
"""
import numpy as np
import pytest

from conftest import rel_l2
from easybem_b200 import meshes

pytestmark = pytest.mark.gpu

FP64_TOL, MIXED_TOL = 1e-12, 1e-6


def pole_graded_sphere(n=64, ratio=0.9, north=90, south=20):
    """Rings of n vertices whose distance to the poles shrinks by ratio, closed by fans."""
    theta = 0.5 * np.pi * ratio ** np.abs(np.arange(-north, south + 1))
    theta[north + 1:] = np.pi - theta[north + 1:]
    rings, phi = len(theta), 2 * np.pi * np.arange(n) / n
    nodes = np.stack([np.outer(np.sin(theta), np.cos(phi)), np.outer(np.sin(theta), np.sin(phi)),
                      np.outer(np.cos(theta), np.ones(n))], -1).reshape(-1, 3)
    i, j = (x.ravel() for x in np.meshgrid(np.arange(rings - 1), np.arange(n), indexing="ij"))
    k = (j + 1) % n
    a, b, c, d = i * n + j, i * n + k, (i + 1) * n + k, (i + 1) * n + j
    j, k = np.arange(n), (np.arange(n) + 1) % n
    top, bottom, last = np.full(n, rings * n), np.full(n, rings * n + 1), (rings - 1) * n
    elems = np.vstack([np.stack(t, 1) for t in ((a, d, c), (a, c, b), (top, j, k), (bottom, last + k, last + j))])
    return np.vstack([nodes, [[0, 0, 1], [0, 0, -1]]]), (elems + 1).astype(np.int32)


def edge_graded_cube(n=40, ratio=0.8):
    """The unit cube with n x n quadrangles a face that shrink by ratio towards its edges."""
    s = np.concatenate([[0], np.cumsum(ratio ** np.arange(n // 2, 0, -1))])
    s = 0.5 * s / s[-1]
    x = np.concatenate([s, 1 - s[-2::-1]])
    grid = np.stack(np.meshgrid(x, x, indexing="ij"), -1)
    i, j = (y.ravel() for y in np.meshgrid(np.arange(n), np.arange(n), indexing="ij"))
    a = i * (n + 1) + j
    quad = np.vstack([np.stack([a, a + n + 1, a + n + 2], 1), np.stack([a, a + n + 2, a + 1], 1)])
    nodes, elems = [], []
    for axis in range(3):
        for side in (0.0, 1.0):
            p = np.empty((n + 1, n + 1, 3))
            p[..., axis], p[..., (axis + 1) % 3], p[..., (axis + 2) % 3] = side, grid[..., 0], grid[..., 1]
            elems.append((quad if side else quad[:, ::-1]) + len(nodes) * (n + 1) ** 2)
            nodes.append(p.reshape(-1, 3))
    nodes = np.vstack(nodes)
    _, first, inverse = np.unique(np.round(nodes * 2.0 ** 40).astype(np.int64), axis=0, return_index=True,
                                  return_inverse=True)
    return nodes[first], (inverse.ravel()[np.vstack(elems)] + 1).astype(np.int32)


def two_spheres(coarse, fine, radius, gap):
    """A unit sphere and, gap beside it, one of the given radius."""
    (v, f), (w, g) = meshes.icosphere(coarse), meshes.icosphere(fine)
    at = (1 + gap + radius) * np.array([0.36, 0.48, 0.8])
    return np.vstack([v, radius * w + at]), np.vstack([f, g + len(v)]).astype(np.int32)


MESHES = {
    "pole": pole_graded_sphere,
    "cube": edge_graded_cube,
    "bodies10": lambda: two_spheres(3, 4, 0.1, 0.5),
    "bodies50": lambda: two_spheres(3, 4, 0.02, 0.2),
    "bodies50_touching": lambda: two_spheres(4, 4, 0.02, 0.01),
}


@pytest.mark.parametrize("name", list(MESHES))
def test_rows_of_the_smallest_triangles(gpu_lib, name):
    nodes, elems = MESHES[name]()
    rng = np.random.default_rng(len(name))
    t, u = rng.normal(size=len(elems)), rng.normal(size=len(nodes))
    p = nodes[elems - 1]
    area = np.linalg.norm(np.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]), axis=1)
    rows = np.argsort(area, kind="stable")[:len(elems) // 4]
    with gpu_lib.Mesh(nodes, elems) as m:
        def apply(engine, prec):
            m.set_far_engine(engine)
            return [x[rows] for x in (*m.apply_sl_dl(t, u, precision=prec), m.apply_sl(t, prec), m.apply_dl(u, prec),
                                      m.dirichlet_rhs(np.stack([u, u[::-1]]), prec)[1])]

        assert m.far_engine("mixed") == "tree" and m.far_engine("fp64") == "tree"
        ref, sym = apply("cuda", "fp64"), apply("sym_all", "fp64")
        rounding = [rel_l2(s, r) for s, r in zip(sym, ref)]
        rounding[3] = rounding[4] = rounding[1]  # the double layer again (the ordered-pair kernels both times)
        for got, r, e in zip(apply("tree", "fp64"), ref, rounding):
            assert rel_l2(got, r) < max(FP64_TOL, 3 * e)
        for got, r in zip(apply("tree", "mixed"), ref):
            assert rel_l2(got, r) < MIXED_TOL


@pytest.mark.parametrize("name", ["sphere", "cube", "bodies10"])
def test_potentials_at_a_probe(gpu_lib, name):
    """Points much closer together than the cells beside them are large, where
    the potential of a rough density nearly cancels: as accurate as the point
    sums in the same precision, within a factor of two."""
    nodes, elems = meshes.perturbed_icosphere(5, seed=3) if name == "sphere" else MESHES[name]()
    rng = np.random.default_rng(7)
    t, u = rng.normal(size=len(elems)), rng.normal(size=len(nodes))
    pts = np.array([1.2, 0.3, 0.1]) + 1e-3 * rng.normal(size=(50000, 3))
    with gpu_lib.Mesh(nodes, elems) as m:
        m.set_far_engine("cuda")
        ref, direct = m.evaluate(pts, t, u, "fp64"), m.evaluate(pts, t, u, "mixed")
        m.set_far_engine("tree")
        assert rel_l2(m.evaluate(pts, t, u, "mixed"), ref) < 2 * rel_l2(direct, ref)
        assert rel_l2(m.evaluate(pts, t, u, "fp64"), ref) < FP64_TOL


@pytest.mark.parametrize("name, north, south, engine", [("small", 25, 5, "sym"), ("third", 30, 8, "tree")])
def test_many_close_cells(gpu_lib, name, north, south, engine):
    """More than a third of the cell pairs close: all of them up to 140 cells
    (3,968 triangles), the tree for larger meshes; against the ordered pairs."""
    nodes, elems = pole_graded_sphere(64, 0.9, north, south)
    rng = np.random.default_rng(north)
    t, u = rng.normal(size=len(elems)), rng.normal(size=len(nodes))
    with gpu_lib.Mesh(nodes, elems) as m:
        assert m.far_engine("fp64") == engine and m.far_engine("mixed") == engine
        got = {prec: m.apply_sl_dl(t, u, precision=prec) for prec in ("fp64", "mixed")}
        m.set_far_engine("cuda")
        v, q = m.apply_sl_dl(t, u)
    for prec, tol in (("fp64", FP64_TOL), ("mixed", MIXED_TOL)):
        assert rel_l2(got[prec][0], v) < tol and rel_l2(got[prec][1], q) < tol
