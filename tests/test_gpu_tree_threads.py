"""Batches and calls on several threads over one mesh, whose lists the first of
them makes: every result is bitwise that of a mesh used by one thread."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from easybem_b200 import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order, n_u", [(4, 40), (4, 140), (9, 140)])
def test_lists_made_by_several_threads(gpu_lib, order, n_u):
    """All cells close, separated clusters, and a rule whose close pairs run in
    forward order. Four batches are made and two host calls run on a new mesh
    at once (batches are applied one after the other: their first apply
    captures a graph)."""
    nodes, elems = meshes.torus(n_u, 0.3)
    rng = np.random.default_rng(n_u)
    t, u, g = rng.normal(size=len(elems)), rng.normal(size=len(nodes)), rng.normal(size=(4, len(nodes)))

    def calls(m, submit):
        batches = [submit(lambda prec=prec: gpu_lib.Batch([m, m], precision=prec, sl_dl=True))
                   for prec in ("mixed", "fp64", "mixed", "fp64")]
        host = [submit(lambda: m.apply_sl_dl(t, u)), submit(lambda: m.dirichlet_rhs(g, "mixed"))]
        size = submit(lambda: [m.near_field_bytes() for _ in range(100)])
        out = [x for h in host for x in h()]
        for b in batches:
            for x in b().apply_sl_dl([t, t], [u, u]):
                out += x
            b().close()
        return out, size()

    def now(fn):
        value = fn()
        return lambda: value

    with gpu_lib.Mesh(nodes, elems, order=order) as m:
        want, size = calls(m, now)
    with ThreadPoolExecutor(7) as pool:
        for _ in range(10):
            with gpu_lib.Mesh(nodes, elems, order=order) as m:
                got, sizes = calls(m, lambda fn: pool.submit(fn).result)
            assert sizes == size and len(got) == len(want)
            assert all(np.array_equal(a, b) for a, b in zip(got, want))
