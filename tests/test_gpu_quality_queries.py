"""Quality queries at the edges of their kernels: histograms of one bin to more than shared memory
holds, meshes of a few elements, flipped elements, and the statistics against the per-element
qualities they summarise."""
import numpy as np
import pytest

from volumesurfacediscretemeshoptimization_b200 import meshgen as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make,jitter", [("tet", 0.3), ("tet", 0.9), ("tri", 0.4), ("hex", 0.3)])
@pytest.mark.parametrize("n", [1, 5, 17])
def test_queries_match_the_element_qualities(vsdmo, make, jitter, n):
    if make == "tri":
        m, cls = vsdmo.DMOMeshTri(*G.tri_grid(n + 2, 1, jitter)), vsdmo.DMOTriFlatClass
    elif make == "tet":
        m, cls = vsdmo.DMOMeshTet(*G.tet_cube(n, 1, jitter)), vsdmo.DMOTetClass
    else:
        m, cls = vsdmo.DMOMeshHex(*G.hex_cube(n, 1, jitter)), vsdmo.DMOHexClass
    opt = cls(m, n_iter=1)
    q = opt.getElementQualities()
    mn, mean = opt.quality_stats()
    assert mn == q.min() and opt.findMinimumQuality() == q.min()
    # the same float values summed in double, in another order
    assert abs(mean - q.astype(np.float64).mean()) <= 1e-12
    for bins in (1, 10, 33, 1024, 1025, 3000):
        x = np.minimum(np.float32(0.9999), q)
        want = np.bincount(np.where(x > 0, (x * np.float32(bins)).astype(np.int32), 0), minlength=bins)
        assert np.array_equal(opt.getQualityHistogram(bins), want), bins
