"""Heat and XSPH in the one-thread forms, which read neighbour attributes by sorted index, against
the FP32 oracle: the water set, the snow set, both or none of them in that form (the water's
committed velocities have to reach the snow's pass either way)."""
import numpy as np
import pytest

from snowsimulation_b200 import scene
from snowsimulation_b200.abi import QUIRKS_FIXED, QUIRKS_REFERENCE
from tests._util import diff_worlds

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("quirks", [QUIRKS_REFERENCE, QUIRKS_FIXED])
@pytest.mark.parametrize("water,snow", [
    ((41, 40, 41), (12, 12, 12)),    # 67,240 | 1,728: the line of XSPH is 65,536
    ((12, 12, 12), (41, 40, 41)),
    ((41, 40, 41), (41, 40, 41)),
    ((32, 32, 32), (32, 32, 32)),    # both below it, heat above its own line
])
def test_attribute_forms_match_oracle(cuda, water, snow, quirks):
    from oracle.oracle import OracleWorld
    from snowsimulation_b200.world import Simulation
    w = scene.scene_drop(water, snow, seed=6, water_jitter=0.003, snow_jitter=0.003, drop_height=0.004, name="attrs")
    rng = np.random.default_rng(4)
    for s in (w.sph, w.dem):
        s["velocity"][:] = rng.uniform(-0.5, 0.5, s["velocity"].shape).astype(np.float32)
    g = Simulation(w, quirks=quirks)
    o = OracleWorld(w, 32, quirks=quirks)
    for _ in range(2):
        g.step()
        o.step()
        assert not diff_worlds(o.w, g.to_host())
