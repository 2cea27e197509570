"""The 8 x 8 flat search with four vertices per warp, bit for bit against the oracle: rings of one to
two rounds of its eight lanes and beyond its limit (the general search), rings of different sizes in
one warp, flipped starts, exact lattices (every key a tie), one to four levels, classes that leave a
warp partly empty, and single meshes whose classes are large enough to take it by themselves."""
import numpy as np
import pytest

from volumesurfacediscretemeshoptimization_b200 import meshgen as G

pytestmark = pytest.mark.gpu
TRI, QUAD = 0, 1


def _star(sectors, m, quads, jitter, seed):
    """Disk of `sectors` patches around a centre vertex of that valence (quads, or triangles)."""
    ids, xy = {}, []

    def vert(s, i, j):
        key = (-1, 0) if i == 0 and j == 0 else ((s % sectors, i) if j == 0 else ((s + 1) % sectors, j) if i == 0 else (s, i, j))
        if key not in ids:
            a = 2 * np.pi * np.array([s, s + 1]) / sectors
            ids[key] = len(xy)
            xy.append(i * np.array([np.cos(a[0]), np.sin(a[0])]) + j * np.array([np.cos(a[1]), np.sin(a[1])]))
        return ids[key]

    q = np.array([[vert(s, i, j), vert(s, i + 1, j), vert(s, i + 1, j + 1), vert(s, i, j + 1)]
                  for s in range(sectors) for i in range(m) for j in range(m)], np.int32)
    xy = np.array(xy) / m
    el = q if quads else np.concatenate([q[:, [0, 1, 3]], q[:, [1, 2, 3]]]).astype(np.int32)
    edges = np.sort(np.concatenate([el[:, [a, (a + 1) % el.shape[1]]] for a in range(el.shape[1])]), 1)
    u, n = np.unique(edges, axis=0, return_counts=True)
    inner = np.ones(len(xy), bool)
    inner[u[n == 1].ravel()] = False
    r = np.random.default_rng(seed).uniform(-jitter / m, jitter / m, xy.shape)
    return np.concatenate([xy + r * inner[:, None], np.zeros((len(xy), 1))], 1).astype(np.float32), el


def _check(oracle_mod, vsdmo, meshes, depth, iters=3):
    b = vsdmo.BatchDMO(meshes)
    b.set_config(8, depth, 8)
    b.iterate(iters)
    for i, (t, xyz, el) in enumerate(meshes):
        om = oracle_mod.OracleMesh(t, xyz, el)
        x = om.xyz
        for _ in range(iters):
            for v0, v1 in om.color_ranges():
                x = om.dmo_flat_f32(x, v0, v1, nq=8, depth=depth)
        got = b.mesh_positions(i)
        assert np.array_equal(got.view(np.uint32), x[om.array(1)].view(np.uint32)), i


@pytest.mark.parametrize("valence", [3, 5, 8, 9, 16, 17])
def test_valences_bitwise(oracle_mod, vsdmo, valence):
    j = 0.3 * min(1.0, 6 / valence)
    meshes = [(TRI, *_star(valence, 4, False, j, 1)), (QUAD, *_star(valence, 4, True, j, 2)), (TRI, *G.tri_grid(7, 3))]
    _check(oracle_mod, vsdmo, meshes, 3)


@pytest.mark.parametrize("depth", [1, 2, 4])
def test_levels_and_flipped_starts_bitwise(oracle_mod, vsdmo, depth):
    meshes = [(TRI, *G.tri_grid(11, 4, 0.9)), (QUAD, *G.quad_grid(12, 5, 0.9)), (TRI, *G.tri_grid(9, None)),
              (QUAD, *G.quad_grid(9, None)), (QUAD, *_star(6, 3, True, 0.5, 6))]
    _check(oracle_mod, vsdmo, meshes, depth, 2)


@pytest.mark.parametrize("kind", [TRI, QUAD])
def test_large_single_mesh_bitwise(oracle_mod, vsdmo, kind):
    xyz, el = (G.tri_grid if kind == TRI else G.quad_grid)(151, 7, 0.4)
    om = oracle_mod.OracleMesh(kind, xyz, el)
    gm = (vsdmo.DMOMeshTri if kind == TRI else vsdmo.DMOMeshQuad)(xyz, el)
    sizes = np.diff(gm.array(vsdmo.A_COL_FREE))
    assert sizes.max() >= 2048 > sizes.min()   # classes on both sides of the rule
    (vsdmo.DMOTriFlatClass if kind == TRI else vsdmo.DMOQuadFlatClass)(gm, n_iter=2).optimize()
    x = om.xyz
    for _ in range(2):
        for v0, v1 in om.color_ranges():
            x = om.dmo_flat_f32(x, v0, v1, nq=8, depth=3)
    assert np.array_equal(gm.positions().view(np.uint32), x.view(np.uint32))
