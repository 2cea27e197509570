"""Tet interior search, bit for bit against the oracle, where the candidate filter and the
split of a key over lanes can go wrong: rings below and above one round of 32 tets and of odd
size, flipped tets (the linear filter), exact lattices (every key a tie), tiny and shifted
coordinates, grids far larger and smaller than the ring, one to eight levels."""
import numpy as np
import pytest

from volumesurfacediscretemeshoptimization_b200 import meshgen as G

pytestmark = pytest.mark.gpu


def _split(xyz, el, share, rounds, seed):
    """1-4 splits at the centre of a share of the tets, repeatedly: valences from 4 to far over 32."""
    r = np.random.default_rng(seed)
    xyz = xyz.astype(np.float64)
    for _ in range(rounds):
        pick = r.random(len(el)) < share
        s = el[pick]
        c = len(xyz) + np.arange(len(s), dtype=np.int32)
        xyz = np.concatenate([xyz, (xyz[s] * r.dirichlet([4] * 4, len(s))[:, :, None]).sum(1)])
        parts = []
        for k in range(4):
            t = s.copy()
            t[:, k] = c
            parts.append(t)
        el = np.concatenate([el[~pick]] + parts).astype(np.int32)
    return xyz.astype(np.float32), el


CASES = {
    "refined": lambda: _split(*G.tet_cube(6, seed=1, jitter=0.15), 0.3, 1, 5),
    "refined_twice": lambda: _split(*G.tet_cube(5, seed=2, jitter=0.1), 0.5, 2, 6),
    "flipped": lambda: G.tet_cube(7, seed=3, jitter=0.9),
    "lattice": lambda: G.tet_cube(6, None),
    "tiny": lambda: (G.tet_cube(5, seed=4)[0] * np.float32(2.0 ** -12), G.tet_cube(5, seed=4)[1]),
    "shifted": lambda: (G.tet_cube(5, seed=6)[0] + np.float32(1000.0), G.tet_cube(5, seed=6)[1]),
}


@pytest.mark.parametrize("name", list(CASES))
def test_runs_bitwise(oracle_mod, vsdmo, name):
    xyz, el = CASES[name]()
    om = oracle_mod.OracleMesh(oracle_mod.TET, xyz, el)
    gm = vsdmo.DMOMeshTet(xyz, el)
    if name.startswith("refined"):
        k = np.diff(gm.array(vsdmo.A_HF_ROWPTR))[gm.info["nSurf"]:]
        assert k.min() == 4 and k.max() > 32
    opt = vsdmo.DMOTetClass(gm, n_iter=4, check_monotone=False)
    opt.optimize()
    ref = om.optimize_f32(om.xyz, 4)[0]
    assert np.array_equal(gm.positions().view(np.uint32), ref.view(np.uint32))


@pytest.mark.parametrize("grid_scale", [1e-3, 3.0, 1e4])
def test_grid_scales_bitwise(oracle_mod, vsdmo, grid_scale):
    xyz, el = G.tet_cube(6, seed=8)
    om = oracle_mod.OracleMesh(oracle_mod.TET, xyz, el)
    gm = vsdmo.DMOMeshTet(xyz, el)
    opt = vsdmo.DMOTetClass(gm, gridScale=grid_scale, n_iter=2, check_monotone=False)
    opt.optimize()
    ref = om.optimize_f32(om.xyz, 2, grid_scale)[0]
    assert np.array_equal(gm.positions().view(np.uint32), ref.view(np.uint32))
