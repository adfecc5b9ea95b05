"""Points of an evaluation through the tree that groups cannot hold, or that
lie far apart, against the direct sums (1e-12 in FP64, 1e-6 mixed)."""
import numpy as np
import pytest

from conftest import rel_l2
from easybem_b200 import meshes

pytestmark = pytest.mark.gpu

PRECISIONS = [("fp64", 1e-12), ("mixed", 1e-6)]


@pytest.fixture(scope="module")
def surface(gpu_lib):
    nodes, elems = meshes.perturbed_icosphere(5, seed=3)
    rng = np.random.default_rng(11)
    with gpu_lib.Mesh(nodes, elems) as m:
        yield m, rng.normal(size=len(elems)), rng.normal(size=len(nodes))


def _inside(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(n, 3))
    return x * 0.6 * rng.uniform(size=(n, 1)) ** (1 / 3) / np.linalg.norm(x, axis=1, keepdims=True)


def _evaluate(surface, pts, prec, engine):
    m, t, u = surface
    m.set_far_engine(engine)
    try:
        return m.evaluate(pts, t, u, prec)
    finally:
        m.set_far_engine("tree")


@pytest.mark.parametrize("prec, tol", PRECISIONS)
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan, 1e200, -1e160])
@pytest.mark.parametrize("count", [1, 40, 20000])
def test_points_out_of_range_leave_the_others_alone(surface, bad, count, prec, tol):
    pts = _inside(20000, 1)
    good = _evaluate(surface, pts, prec, "tree")
    at = np.random.default_rng(count).choice(len(pts), count, replace=False)
    pts[at, np.arange(count) % 3] = bad
    p, d = _evaluate(surface, pts, prec, "tree"), _evaluate(surface, pts, prec, "cuda")
    assert np.allclose(p[at], d[at], rtol=tol, atol=0.0, equal_nan=True)
    rest = np.delete(np.arange(len(pts)), at)
    if len(rest):
        assert np.isfinite(p[rest]).all() and rel_l2(p[rest], good[rest]) < tol
