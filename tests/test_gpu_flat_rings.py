"""The flat triangle search of one vertex per warp on rings around the warp's 32 lanes, launched class after
class with and without a graph, bit for bit against the oracle (one rounding per operation on both
sides, so no tolerance)."""
import numpy as np
import pytest

from volumesurfacediscretemeshoptimization_b200 import meshgen as G

pytestmark = pytest.mark.gpu


def fan(n, seed):
    """A disk: a centre of valence n, two rings of n vertices."""
    a = 2 * np.pi * np.arange(n) / n
    ring = np.stack([np.cos(a), np.sin(a)], 1)
    xy = np.concatenate([np.zeros((1, 2)), 0.5 * ring, ring])
    r = np.random.default_rng(seed).uniform(-0.3, 0.3, xy.shape) * min(0.5, 1.5 / n)
    r[n + 1:] = 0
    j, k = np.arange(n), (np.arange(n) + 1) % n
    el = np.concatenate([np.stack([0 * j, 1 + j, 1 + k], 1), np.stack([1 + j, 1 + n + j, 1 + n + k], 1),
                         np.stack([1 + j, 1 + n + k, 1 + k], 1)])
    return np.concatenate([xy + r, np.zeros((len(xy), 1))], 1).astype(np.float32), el.astype(np.int32)


@pytest.mark.parametrize("use_graph", [True, False])
@pytest.mark.parametrize("valence", [3, 31, 32, 33, 65, 0])
def test_rings_bitwise(oracle_mod, vsdmo, valence, use_graph):
    xyz, el = fan(valence, 1) if valence else G.tri_grid(40, 3)
    om = oracle_mod.OracleMesh(0, xyz, el)
    gm = vsdmo.DMOMeshTri(xyz, el)
    vsdmo.DMOTriFlatClass(gm, n_iter=4, use_graph=use_graph).optimize()
    x = om.xyz
    for _ in range(4):
        for v0, v1 in om.color_ranges():
            x = om.dmo_flat_f32(x, v0, v1, nq=8, depth=3)
    assert np.array_equal(gm.positions().view(np.uint32), x.view(np.uint32))
