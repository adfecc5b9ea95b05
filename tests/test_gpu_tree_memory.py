"""Partial slots of the tree far field: bounded, as the symmetric kernels' are."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def needles(ne, length):
    """ne separate needles in the unit cube: their cells are as large as they are long."""
    rng = np.random.default_rng(0)
    c, d = rng.uniform(0, 1, size=(ne, 1, 3)), rng.normal(size=(ne, 1, 3))
    d *= 0.5 * length / np.linalg.norm(d, axis=2, keepdims=True)
    nodes = np.concatenate([c - d, c + d, c + 0.01 * rng.normal(size=(ne, 1, 3))], axis=1).reshape(-1, 3)
    return nodes, (np.arange(3 * ne).reshape(-1, 3) + 1).astype(np.int32)


def test_meshes_with_too_many_close_cells_keep_the_direct_kernels(gpu_lib):
    """A quarter of all cell pairs close: below the share that ends the tree,
    but 46 GiB of slots in SL+DL (32 GiB are the limit; the symmetric kernels
    end at 524,288 triangles)."""
    with gpu_lib.Mesh(*needles(800_000, 0.26)) as m:
        assert m.far_engine("mixed") == "cuda" and m.far_engine("fp64") == "cuda"
    nodes, elems = needles(60_000, 0.2)
    with gpu_lib.Mesh(nodes, elems) as m:
        assert m.far_engine("mixed") == "tree" and m.far_engine("fp64") == "tree"
