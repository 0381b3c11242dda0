"""Density passes that take the snow's own sums from lists with a skin, against the FP32 oracle:
snow that stays within the skin, that leaves it inside its cells, that changes cells, and lists
that overflow through the skin's candidates only; with water beside it, links forming."""
import numpy as np
import pytest

from snowsimulation_b200 import scene
from snowsimulation_b200.abi import QUIRKS_FIXED, QUIRKS_REFERENCE
from tests._util import diff_worlds

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("quirks", [QUIRKS_REFERENCE, QUIRKS_FIXED])
@pytest.mark.parametrize("spacing,speed", [(0.02, 0.0), (0.02, 0.02), (0.02, 0.15), (0.02, 2.0), (0.009, 0.02)])
def test_skin_lists_match_oracle(cuda, spacing, speed, quirks):
    from oracle.oracle import OracleWorld
    from snowsimulation_b200.world import Simulation
    w = scene.scene_drop((8, 4, 8), (36, 34, 36), seed=8, spacing=spacing, water_jitter=0.05 * spacing,
                         snow_jitter=0.05 * spacing, drop_height=0.004, init_links=True, name="skin")
    v = w.dem["velocity"]
    v[:] = np.random.default_rng(5).uniform(-speed, speed, v.shape).astype(np.float32)
    g = Simulation(w, quirks=quirks)
    o = OracleWorld(w, 32, quirks=quirks)
    for n in (1, 3):
        g.step(substeps=n)
        for _ in range(n):
            o.step()
        assert not diff_worlds(o.w, g.to_host())
