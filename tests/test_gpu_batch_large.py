"""Batched scenes above every line between the forms of the substep's passes (sets whose sizes
together take one thread a particle, the snow's lists with a skin and the neighbour attributes by
sorted index, all with scene ids): every scene equals the same scene run alone, bit for bit.  Alone
each is below the lines (one warp a particle), so the two runs share no form of those passes."""
import ctypes as C

import numpy as np
import pytest

from snowsimulation_b200 import scene
from snowsimulation_b200.batch import BatchSimulation
from tests.test_gpu_batch import _alone, _compare

pytestmark = pytest.mark.gpu
SORTS_FULL_DEM, SORTS_KEPT_DEM, SKIN_PASSES, SKIN_WALKS = 21, 23, 24, 25    # of snowb_device_counters


def _scenes(moving):
    """Five scenes of 9,000 to 18,816 snow particles (75,424 together).  At rest under water that
    is still falling (two of the blocks, 27,816 particles, a plain lattice); or moving: one scene with snow that changes cells in every substep, one
    that freezes and melts, water between the snow of the others."""
    drop = 0.004 if moving else 0.2
    ws = [scene.scene_drop(water, snow, seed=11 + k, water_jitter=0.002, drop_height=drop,
                           snow_jitter=0.002 if moving or k % 3 else 0.0, init_links=True)
          for k, (water, snow) in enumerate([((8, 4, 8), (28, 24, 28)), ((3, 5, 7), (30, 20, 30)), ((6, 6, 6), (26, 24, 26)),
                                             ((10, 10, 10), (30, 10, 30)), ((2, 2, 2), (28, 18, 36))])]
    if moving:
        v = ws[1].dem["velocity"]
        v[:] = np.random.default_rng(3).uniform(-2, 2, v.shape).astype(np.float32)
        w = ws[2]
        w.sph["T"][: w.n_sph // 2] = -1.0
        w.sph["new_T"][:] = w.sph["T"]
        w.dem["T"][:300] = 2.0
        w.dem["new_T"][:] = w.dem["T"]
    return ws


@pytest.mark.parametrize("moving", [False, True])
def test_large_batch_equals_independent(cuda, moving):
    worlds = _scenes(moving)
    substeps = 5
    alone = [_alone(w, substeps, True) for w in worlds]
    b = BatchSimulation(worlds).setup()
    assert b.n_dem > 65536 and max(w.n_sph + w.n_dem for w in worlds) < 40000
    b.step(substeps=substeps, use_graph=True)
    n = (C.c_uint32 * 27)()
    assert b.lib.snowb_device_counters(n, 27) == 0
    if moving:     # a moving scene takes the whole set's sort along
        assert n[SORTS_FULL_DEM] > n[SORTS_KEPT_DEM]
    else:
        assert n[SORTS_KEPT_DEM] > n[SORTS_FULL_DEM]
        assert n[SKIN_PASSES] * b.n_dem - n[SKIN_WALKS] > n[SKIN_PASSES] * 9000 > 0   # the lists with a skin serve
    bw, sid = b.to_host()
    _compare(worlds, bw, sid, alone)
