"""Searches on rings where the ring fold of keys is not an ordinary minimum: coincident ring points (0 / 0 at
a candidate that falls on them), points that nearly coincide, NaN positions. Bit for bit against the oracle
(the same operations in the same order on both sides, so no tolerance)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TRI, QUAD, TET, HEX = range(4)


def _fan(n):
    """A disk: a centre of valence n and its ring."""
    a = 2 * np.pi * np.arange(n) / n
    xyz = np.stack([np.cos(a), np.sin(a), 0 * a], 1)
    j = np.arange(n)
    el = np.stack([0 * j, 1 + j, 1 + (j + 1) % n], 1)
    return np.concatenate([np.zeros((1, 3)), xyz]).astype(np.float32), el.astype(np.int32)


def _ring_of(oracle_mod, om, v=0):
    """Ring vertices of v in fan order (the order of its elements)."""
    rp, he = om.array(oracle_mod.A_HE_ROWPTR), om.array(oracle_mod.A_HALFEDGES).reshape(-1, 4)
    return he[rp[v]:rp[v + 1], 0]


@pytest.mark.parametrize("use_graph", [True, False])
def test_nan_key_on_one_lane(oracle_mod, vsdmo, use_graph):
    """The first ring element has no length and the candidate (+S, -S) lies on it: a NaN key on one lane of a
    level at which the others move."""
    xyz, el = _fan(6)
    om = oracle_mod.OracleMesh(TRI, xyz, el)
    gm = vsdmo.DMOMeshTri(xyz, el)
    x = om.xyz.copy()
    ring = _ring_of(oracle_mod, om)
    # the origin lies outside of the ring's kernel (a negative key), those with x > 0.25 do not
    x[ring] = np.array([[0.5, -0.5, 0], [0.5, -0.5, 0], [1, 0.5, 0], [1, 1, 0], [0.25, 1, 0], [0.25, -1, 0]], np.float32)
    x[0] = 0
    opt = vsdmo.DMOTriFlatClass(gm, n_iter=1, use_graph=use_graph, check_monotone=False)
    gm.set_positions(x)
    opt.restart()
    opt.iterate(1)
    want = om.dmo_flat_f32(x, 0, 1, nq=8, depth=3)
    assert not np.array_equal(want[0], x[0])   # it moves
    assert np.array_equal(gm.positions().view(np.uint32), want.view(np.uint32))
