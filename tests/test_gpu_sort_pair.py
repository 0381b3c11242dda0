"""The substep's sorts of both sets in shared launches, and the cell scan that leaves empty chunks
out, against the FP32 oracle: cell tables compared in full, stale entries included.  Grids from one
scan chunk to more than the two-level prefix starts at, empty sets, sets that straddle a warp."""
import numpy as np
import pytest

from snowsimulation_b200 import scene
from snowsimulation_b200.abi import QUIRKS_FIXED, QUIRKS_REFERENCE
from snowsimulation_b200.params import make_sim_params
from tests._util import diff_worlds

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("quirks", [QUIRKS_REFERENCE, QUIRKS_FIXED])
@pytest.mark.parametrize("grid,water,snow", [
    ((8, 8, 8), (3, 2, 3), (4, 2, 4)),          # 512 cells: less than one scan chunk
    ((16, 16, 16), (5, 1, 9), (3, 3, 5)),       # 4 chunks, sizes that straddle a warp
    ((64, 64, 64), (4, 4, 4), (7, 5, 7)),       # 256 chunks, nearly all empty
    ((128, 128, 128), (3, 3, 3), (6, 4, 6)),    # 2,048 chunks: the two-level prefix
])
def test_sorts_match_oracle(cuda, grid, water, snow, quirks):
    from oracle.oracle import OracleWorld
    from snowsimulation_b200.world import Simulation
    p = make_sim_params(grid_size=grid)
    box = scene.boundary_box(0.01)
    box = box[np.abs(box).max(axis=1) < 0.3]     # a patch of floor keeps the small grids' cells small
    w = scene.scene_drop(water, snow, seed=2, water_jitter=0.002, snow_jitter=0.002, drop_height=0.03, params=p,
                         boundary=box, init_links=True, name="sorts")
    w.sph["velocity"][:w.n_sph] = np.random.default_rng(1).uniform(-3, 3, (w.n_sph, 3)).astype(np.float32)
    g = Simulation(w, quirks=quirks).setup()
    o = OracleWorld(w, 32, quirks=quirks).setup()
    for k in range(4):      # calls of one substep, then calls of several (kept sorts among them)
        n = 1 if k < 2 else 3
        g.step(substeps=n)
        for _ in range(n):
            o.step()
        assert not diff_worlds(o.w, g.to_host())
    w2 = g.to_host()        # a caller may write the tables between calls: the next sort clears them
    for cd in (g.scd, g.dcd):
        cd.t["cell_start"].fill_(5)
    for cd in (o.w.sph_cd, o.w.dem_cd):
        cd["cell_start"][:] = 5
    if quirks == QUIRKS_FIXED:
        g.step()
        o.step()
        assert not diff_worlds(o.w, g.to_host())
    assert w2.n_sph + w2.n_dem == w.n_sph + w.n_dem
