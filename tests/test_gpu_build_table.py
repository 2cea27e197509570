"""The connectivity build through the vertex-to-element table: waiting lists, colours in any
order, boundary faces by row. Whole numbers throughout, so every array equals the oracle's."""
import numpy as np
import pytest

from volumesurfacediscretemeshoptimization_b200 import meshgen as G

pytestmark = pytest.mark.gpu


def one_tet(n):
    """n tets around the edge (0, 1): rows of n elements, n = 1 a single tet."""
    a = np.linspace(0, 1.5 * np.pi, n + 1)
    xyz = [(0, 0, 0), (0, 0, 1)] + [(np.cos(t), np.sin(t), 0.5) for t in a]
    return np.array(xyz, np.float32), np.array([(0, 1, 2 + i, 3 + i) for i in range(n)], np.int32)


MESHES = {
    "tet1": ("DMOMeshTet", 2, lambda: one_tet(1)),
    "tet31": ("DMOMeshTet", 2, lambda: one_tet(31)),
    "tet33": ("DMOMeshTet", 2, lambda: one_tet(33)),
    "tet53": ("DMOMeshTet", 2, lambda: one_tet(53)),     # 159 faces in row 0, of 160 that the shared list holds
    "tet54": ("DMOMeshTet", 2, lambda: one_tet(54)),     # 162: the spilled list
    "cube5": ("DMOMeshTet", 2, lambda: G.tet_cube(5)),
    "hex4": ("DMOMeshHex", 3, lambda: G.hex_cube(4)),
    "tri9": ("DMOMeshTri", 0, lambda: G.tri_grid(9, 7)),
    "quad9": ("DMOMeshQuad", 1, lambda: G.quad_grid(9, 7)),
}


@pytest.mark.parametrize("seed", ["1", "77", "reference", "rounds"])
@pytest.mark.parametrize("name", list(MESHES))
def test_every_array_equals_the_oracle(oracle_mod, vsdmo, name, seed):
    cls, kind, gen = MESHES[name]
    seed = {"reference": vsdmo.COLOR_REFERENCE, "rounds": vsdmo.COLOR_ROUNDS | 3}.get(seed) or int(seed)
    xyz, el = gen()
    gm = getattr(vsdmo, cls)(xyz, el, color_seed=seed)
    om = oracle_mod.OracleMesh(kind, xyz, el, color_seed=seed)
    assert om.info == gm.info
    A, B = om.arrays(), gm.arrays()
    for k in A:
        if A[k].dtype == np.float32:
            assert np.array_equal(A[k].view(np.uint32) & 0x7fffffff, B[k].view(np.uint32) & 0x7fffffff) or \
                np.array_equal(A[k], B[k], equal_nan=True), k
        else:
            assert np.array_equal(A[k], B[k]), k
