"""The batch's general search: its resident blocks where no mesh is on the packed search (four blocks of 256 threads
per SM whatever the ring, as its shared memory is a quarter of the packed one's), and its lane widths."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TRI = 0


def _fan(n):
    a = 2 * np.pi * np.arange(n) / n
    j = np.arange(n)
    return (np.concatenate([np.zeros((1, 3)), np.stack([np.cos(a), np.sin(a), 0 * a], 1)]).astype(np.float32),
            np.stack([0 * j, 1 + j, 1 + (j + 1) % n], 1).astype(np.int32))


@pytest.mark.parametrize("valence", [6, 11, 12, 16, 17])
def test_general_search_keeps_its_blocks(vsdmo, valence):
    import torch
    b = vsdmo.BatchDMO([(TRI, *_fan(valence))])
    b.set_config(4, 2, 32)
    b.iterate(1)
    assert b.info()["max_halfedges"] == valence
    assert b.info()["blocks"] == 4 * torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("lanes", [8, 16, 32])
def test_general_search_lanes_bitwise(oracle_mod, vsdmo, lanes):
    """8 x 8 grids on the general search, which a ring of 17 brings to the whole batch, at each lane width."""
    from volumesurfacediscretemeshoptimization_b200 import meshgen as G
    meshes = [(TRI, *_fan(17)), (TRI, *G.tri_grid(20, 1)), (1, *G.quad_grid(15, 2))]
    b = vsdmo.BatchDMO(meshes)
    b.set_config(8, 3, lanes)
    b.iterate(2)
    for i, (t, xyz, el) in enumerate(meshes):
        om = oracle_mod.OracleMesh(t, xyz, el)
        x = om.xyz
        for _ in range(2):
            for v0, v1 in om.color_ranges():
                x = om.dmo_flat_f32(x, v0, v1, nq=8, depth=3)
        assert np.array_equal(b.mesh_positions(i).view(np.uint32), x[om.array(oracle_mod.A_NEW_OF_OLD)].view(np.uint32)), i
