"""Batched flat search with work items of one to several warp steps: every mesh of the batch equals
its own single-mesh run bit for bit (each vertex sees the same positions in both, so no tolerance)."""
import numpy as np
import pytest

from volumesurfacediscretemeshoptimization_b200 import meshgen as G

pytestmark = pytest.mark.gpu


# items of one step (a few hundred vertices a class), and of two (classes of 43,000 over the batch)
@pytest.mark.parametrize("sizes", [(9, 31, 20), (221,) * 4 + (230,) * 3])
def test_batch_equals_single_meshes(vsdmo, sizes):
    meshes = [(i % 2, *(G.quad_grid if i % 2 else G.tri_grid)(n, i + 1)) for i, n in enumerate(sizes)]
    b = vsdmo.BatchDMO(meshes)
    b.iterate(2)
    for i, (kind, xyz, el) in enumerate(meshes):
        gm = (vsdmo.DMOMeshQuad if kind else vsdmo.DMOMeshTri)(xyz, el)
        (vsdmo.DMOQuadFlatClass if kind else vsdmo.DMOTriFlatClass)(gm, n_iter=2).optimize()
        want = gm.positions(original_order=True)
        assert np.array_equal(b.mesh_positions(i).view(np.uint32), want.view(np.uint32)), i
