"""Both forms of the density and lambda pass against the FP32 oracle: set sizes on either side
of the line between them, cells of more than 32 members, neighbour lists that overflow,
boundary particles with and without water or snow around them, an empty boundary."""
import numpy as np
import pytest

from snowsimulation_b200 import scene
from snowsimulation_b200.abi import QUIRKS_FIXED, QUIRKS_REFERENCE
from tests._util import diff_worlds

pytestmark = pytest.mark.gpu

SCENES = {
    "one warp, small": dict(water=(3, 3, 3), snow=(5, 3, 5)),
    "one warp, cells of 60, lists of 300": dict(water=(4, 4, 4), snow=(9, 9, 9), spacing=0.0103),
    "one warp, lists overflow": dict(water=(2, 2, 2), snow=(9, 9, 9), spacing=0.0077),
    "below the line": dict(water=(5, 5, 5), snow=(34, 34, 34)),
    "above the line": dict(water=(5, 5, 5), snow=(35, 34, 34)),
    "no boundary": dict(water=(3, 3, 3), snow=(5, 3, 5), boundary=np.zeros((0, 3), np.float32)),
}


@pytest.mark.parametrize("quirks", [QUIRKS_REFERENCE, QUIRKS_FIXED])
@pytest.mark.parametrize("name", sorted(SCENES))
def test_density_forms_match_oracle(cuda, name, quirks):
    from oracle.oracle import OracleWorld
    from snowsimulation_b200.world import Simulation
    kw = dict(SCENES[name])
    s = kw.pop("spacing", 0.02)
    w = scene.scene_drop(kw.pop("water"), kw.pop("snow"), seed=5, spacing=s, water_jitter=0.1 * s,
                         snow_jitter=0.1 * s, drop_height=0.012, name=name, **kw)
    g = Simulation(w, quirks=quirks)
    o = OracleWorld(w, 32, quirks=quirks)
    if w.n_b:   # the set-up calls refuse an empty boundary's null arrays; a step takes it
        g.setup()
        o.setup()
    for _ in range(2):
        g.step()
        o.step()
        assert not diff_worlds(o.w, g.to_host())
