"""Which particles the snow's lists with a skin serve: the branch that each case of the lists is
there for is the one that runs, by the counters of the density passes and sort points (the results
are the traversal's either way)."""
import ctypes as C

import numpy as np
import pytest

from snowsimulation_b200 import scene
from snowsimulation_b200.abi import QUIRKS_FIXED, QUIRKS_REFERENCE

pytestmark = pytest.mark.gpu
KEPT_DEM, PASSES, WALKS, MARKS = 23, 24, 25, 26     # of snowb_device_counters


@pytest.mark.parametrize("quirks", [QUIRKS_REFERENCE, QUIRKS_FIXED])
@pytest.mark.parametrize("spacing,speed", [(0.02, 0.0), (0.02, 0.15), (0.02, 6.0), (0.009, 0.0)])
def test_skin_lists_serve_what_they_are_for(cuda, spacing, speed, quirks):
    from snowsimulation_b200.world import Simulation
    jitter = 0.05 * spacing if speed else 0.0
    w = scene.scene_drop((8, 4, 8), (36, 34, 36), seed=8, spacing=spacing, water_jitter=jitter, snow_jitter=jitter,
                         drop_height=0.05, init_links=True, name="skin")     # no water within reach
    v = w.dem["velocity"]
    v[:] = np.random.default_rng(5).uniform(-speed, speed, v.shape).astype(np.float32)
    g = Simulation(w, quirks=quirks)
    # the dense block flies apart in the first iteration: up to its density pass only
    g.step(stop_after=12 if spacing == 0.009 else 0)
    c = (C.c_uint32 * 27)()
    assert g.lib.snowb_device_counters(c, 27) == 0
    if speed == 6.0:            # 25 mm a substep in cells of 40 mm: sorted in full after every move
        assert (c[PASSES], c[WALKS], c[MARKS]) == (0, 0, 0)
        return
    if spacing == 0.009:        # 364 neighbours within h, 388 within the skin: past a list's 384
        assert (c[PASSES], c[MARKS]) == (1, 0) and c[WALKS] > g.n_dem // 4
        return
    assert c[KEPT_DEM] > 0 and c[PASSES] > 0
    if speed == 0.0:            # a lattice at rest sinks by 0.17 mm, half the skin is 0.4 mm: all are served
        assert (c[WALKS], c[MARKS]) == (0, 0)
    else:                       # up to 0.6 mm along each axis
        assert c[MARKS] > g.n_dem // 4 and c[WALKS] > 0
