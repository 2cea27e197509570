"""Hex interior search, bit for bit against the oracle, where the candidate filter, the constant key
and the item subset can go wrong: rings of 6 to 64 halfhexes, flipped starts (keys of zero), exact
lattices (every key a tie), many iterations (boxes shrink to rounding size), coordinates so small
that the metric's lower limits decide, grids far larger and smaller than the ring."""
import numpy as np
import pytest

from volumesurfacediscretemeshoptimization_b200 import meshgen as G

pytestmark = pytest.mark.gpu


def _star(sectors, m, layers, jitter, seed):
    """A disk of `sectors` quad patches around a centre vertex, extruded: the centre line has
    2 * sectors halfhexes per interior vertex."""
    ids, xy = {}, []

    def vert(s, i, j):
        key = (-1, 0) if i == 0 and j == 0 else ((s % sectors, i) if j == 0 else ((s + 1) % sectors, j) if i == 0 else (s, i, j))
        if key not in ids:
            a = 2 * np.pi * np.array([s, s + 1]) / sectors
            ids[key] = len(xy)
            xy.append(i * np.array([np.cos(a[0]), np.sin(a[0])]) + j * np.array([np.cos(a[1]), np.sin(a[1])]))
        return ids[key]

    quads = [[vert(s, i, j), vert(s, i + 1, j), vert(s, i + 1, j + 1), vert(s, i, j + 1)]
             for s in range(sectors) for i in range(m) for j in range(m)]
    xy = np.array(xy) / m
    n = len(xy)
    xyz = np.concatenate([np.concatenate([xy, np.full((n, 1), z / m)], 1) for z in range(layers + 1)])
    q = np.array(quads)
    hexes = np.concatenate([np.concatenate([q + (z + 1) * n, q + z * n], 1) for z in range(layers)]).astype(np.int32)
    cnt = np.bincount(hexes.ravel(), minlength=len(xyz))
    rim = np.bincount(q.ravel(), minlength=n)
    inner2 = np.array([rim[i] >= 3 and np.linalg.norm(xy[i]) < 0.99 for i in range(n)])
    inner = np.concatenate([inner2 if 0 < z < layers else np.zeros(n, bool) for z in range(layers + 1)]) & (cnt >= 6)
    r = np.random.default_rng(seed).uniform(-jitter / m, jitter / m, (len(xyz), 3))
    return (xyz + r * inner[:, None]).astype(np.float32), hexes


def _cube(n, jitter, scale=1.0, seed=1):
    x, e = G.hex_cube(n, seed, jitter)
    return (x * np.float32(scale)).astype(np.float32), e


CASES = {
    "star3": (lambda: _star(3, 3, 4, 0.1, 1), 3),
    "star5": (lambda: _star(5, 3, 4, 0.1, 2), 3),
    "star16": (lambda: _star(16, 2, 3, 0.02, 3), 3),
    "star32": (lambda: _star(32, 2, 3, 0.01, 4), 2),
    "flipped": (lambda: _cube(6, 0.9), 3),
    "lattice": (lambda: _cube(5, 0.0), 2),
    "many_iterations": (lambda: _cube(7, 0.3, seed=5), 14),
    "small": (lambda: _cube(6, 0.3, 2.0 ** -4), 3),
    "below_limits": (lambda: _cube(6, 0.3, 2.0 ** -6), 2),
    "large": (lambda: _cube(6, 0.3, 1e4), 3),
}


@pytest.mark.parametrize("name", list(CASES))
def test_runs_bitwise(oracle_mod, vsdmo, name):
    make, iters = CASES[name]
    xyz, el = make()
    om = oracle_mod.OracleMesh(oracle_mod.HEX, xyz, el)
    gm = vsdmo.DMOMeshHex(xyz, el)
    if name.startswith("star"):
        assert 2 * int(name[4:]) in np.diff(gm.array(vsdmo.A_HF_ROWPTR))[gm.info["nSurf"]:]
    opt = vsdmo.DMOHexClass(gm, n_iter=iters, check_monotone=False)
    opt.optimize()
    ref = om.optimize_f32(om.xyz, iters)[0]
    assert np.array_equal(gm.positions().view(np.uint32), ref.view(np.uint32))


@pytest.mark.parametrize("grid_scale", [1e-4, 4.0, 1e3])
def test_grid_scales_bitwise(oracle_mod, vsdmo, grid_scale):
    xyz, el = _cube(6, 0.3, seed=8)
    om = oracle_mod.OracleMesh(oracle_mod.HEX, xyz, el)
    gm = vsdmo.DMOMeshHex(xyz, el)
    opt = vsdmo.DMOHexClass(gm, gridScale=grid_scale, n_iter=3, check_monotone=False)
    opt.optimize()
    ref = om.optimize_f32(om.xyz, 3, grid_scale)[0]
    assert np.array_equal(gm.positions().view(np.uint32), ref.view(np.uint32))
