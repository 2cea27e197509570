"""The batch's autotuner: what it leaves behind when a trial fails."""
import numpy as np
import pytest

from volumesurfacediscretemeshoptimization_b200 import meshgen as G

pytestmark = pytest.mark.gpu
TRI, QUAD = 0, 1
E_TIMEOUT = 6


def test_failed_trial_leaves_the_batch_as_it_was(vsdmo):
    meshes = [(TRI, *G.tri_grid(30, 1)), (TRI, *G.tri_grid(140, 2)), (QUAD, *G.quad_grid(120, 3))]
    config = ([8, 4, 4], [3, 2, 3], [32, 16, 8])
    b = vsdmo.BatchDMO(meshes)
    b.set_config(*config)
    b.iterate(1)
    x = b.positions()
    try:
        vsdmo.debug_set_wait_limit_ns(0)
        with pytest.raises(vsdmo.VSDMOError) as e:
            b.autotune(2)
        assert e.value.status == E_TIMEOUT
    finally:
        vsdmo.debug_set_wait_limit_ns(-1)
    assert all(np.array_equal(a, c) for a, c in zip(b.config(), config))
    assert np.array_equal(b.positions(), x)
    b.iterate(2)
    fresh = vsdmo.BatchDMO(meshes)
    fresh.set_config(*config)
    fresh.iterate(3)
    assert np.array_equal(b.positions(), fresh.positions())


def test_lanes_are_tried_only_where_the_search_has_them(vsdmo):
    """8 x 8 grids with rings of up to 16 run eight lanes per vertex whatever is configured: trials that differ in
    lanes alone would be the same search, and the choice among them noise."""
    meshes = [(TRI, *G.tri_grid(n, n)) for n in (20, 30, 40)] + [(QUAD, *G.quad_grid(n, n)) for n in (60, 70, 80, 110, 120)]
    for repeat in range(3):
        b = vsdmo.BatchDMO(meshes)
        report = b.autotune(2)
        n, depth, lanes = b.config()
        assert np.all(lanes[n == 8] == 32), report
        b.close()
