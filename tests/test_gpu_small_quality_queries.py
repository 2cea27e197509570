"""Minimum and mean quality of small meshes: read back and summed in element order, the shorter way there."""
import numpy as np
import pytest

from volumesurfacediscretemeshoptimization_b200 import meshgen as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 5, 8])
def test_small_mesh_mean_is_the_sequential_sum(vsdmo, n):
    mesh = vsdmo.DMOMeshTet(*G.tet_cube(n, n))
    opt = vsdmo.DMOTetClass(mesh)
    q = opt.getElementQualities()
    low, mean = opt.quality_stats()
    assert low == q.min()
    assert mean == np.add.accumulate(q.astype(np.float64))[-1] / len(q)
