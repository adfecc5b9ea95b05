"""Four double layers at once (right-hand sides) on small meshes: on both sides
of the numbers of cells up to which the tree sums all pairs, above which they
are the direct kernels bit for bit."""
import numpy as np
import pytest

from conftest import rel_l2
from easybem_b200 import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ne, mixed_direct, fp64_direct", [(1024, False, False), (1025, True, False),
                                                           (2880, True, False), (2881, True, True), (3200, True, True)])
def test_right_hand_sides_of_small_meshes(gpu_lib, ne, mixed_direct, fp64_direct):
    nodes, elems = meshes.torus(80, 0.4)
    elems = elems[:ne]
    g = np.random.default_rng(ne).normal(size=(6, len(nodes)))
    with gpu_lib.Mesh(nodes, elems) as m:
        assert m.far_engine("fp64") == "sym"
        for prec, direct, tol in (("mixed", mixed_direct, 1e-6), ("fp64", fp64_direct, 1e-12)):
            m.set_far_engine("tree")
            b = m.dirichlet_rhs(g, prec)
            m.set_far_engine("cuda")
            c = m.dirichlet_rhs(g, prec)
            assert np.array_equal(b, c) == direct
            for x, y in zip(b, c):
                assert rel_l2(x, y) < tol
