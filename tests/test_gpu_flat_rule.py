"""The size from which a single flat mesh is searched four vertices per warp: not where that is the longer chain."""
import time

import pytest

from volumesurfacediscretemeshoptimization_b200 import meshgen as G

pytestmark = pytest.mark.gpu


def test_first_iteration_grows_with_the_mesh_only(vsdmo):
    """One iteration from a jittered start, latency bound at both sizes: classes of up to 2,700 vertices against
    1,800. 1.1 times as long with a warp per vertex, 1.9 with four vertices per warp."""
    import torch
    times = []
    for n in (90, 110):
        mesh = vsdmo.DMOMeshTri(*G.tri_grid(n, 1, 0.4))
        opt = vsdmo.DMOTriFlatClass(mesh, n_iter=1, check_monotone=False)
        x = mesh.positions()
        best = 1e9
        for _ in range(40):
            mesh.set_positions(x)
            opt.restart()
            torch.cuda.synchronize()
            t = time.perf_counter()
            opt.iterate(1)
            best = min(best, time.perf_counter() - t)
        times.append(best)
    assert times[1] < 1.5 * times[0], times
