"""The triangle surface search with two candidates per lane packed: fans of every size around
its chunks (the ring key at the start position folds 32 triangles at a time) against the CPU
oracle, bit for bit (every operation has one rounding on both sides, so no tolerance)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def smooth_cap_sphere(valence, rings=12, seed=0):
    """A sphere whose two poles have ``valence`` neighbours, jittered tangentially."""
    v = [(0.0, 0.0, 1.0)]
    for r in range(1, rings):
        t = np.pi * r / rings
        for j in range(valence):
            p = 2 * np.pi * (j + 0.5 * (r & 1)) / valence
            v.append((np.sin(t) * np.cos(p), np.sin(t) * np.sin(p), np.cos(t)))
    v.append((0.0, 0.0, -1.0))
    f = []
    at = lambda r, j: 1 + (r - 1) * valence + j % valence
    for j in range(valence):
        f.append((0, at(1, j), at(1, j + 1)))
        f.append((len(v) - 1, at(rings - 1, j + 1), at(rings - 1, j)))
        for r in range(1, rings - 1):
            o = r & 1
            f.append((at(r, j), at(r + 1, j + o), at(r, j + 1)))
            f.append((at(r + 1, j + o), at(r + 1, j + o + 1), at(r, j + 1)))
    v = np.array(v) + np.random.default_rng(seed).uniform(-1, 1, (len(v), 3)) * (0.15 / max(rings, valence))
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    return v.astype(np.float32), np.array(f, np.int32)


@pytest.mark.parametrize("valence", [19, 24, 31, 32, 33, 63])
def test_fans_of_every_chunk_size_bitwise(oracle_mod, vsdmo, valence):
    xyz, el = smooth_cap_sphere(valence, rings=max(12, valence // 2))
    om = oracle_mod.OracleMesh(0, xyz, el)
    gm = vsdmo.DMOMeshTri(xyz, el)
    assert gm.info == om.info
    opt = vsdmo.DMOTriClass(gm, n_iter=3)
    if om.info["nFeature"]:
        pytest.skip("feature edges on this sphere")
    state = om.surface_state_f32(om.xyz)
    x, moved = om.xyz, 0
    for c, (v0, v1) in enumerate(om.color_ranges()):
        y = om.dmo_surf_color_f32(x, state, v0, v1)
        moved += int(np.any(y != x, axis=1).sum())
        x = y
        opt.run_color(c)
        g = gm.positions()
        same = (g.view(np.uint32) == x.view(np.uint32)) | (np.isnan(g) & np.isnan(x))
        assert same.all(), (c, np.argwhere(~same)[:4])
    assert moved > 0
