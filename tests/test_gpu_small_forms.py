"""The one-warp-per-particle forms of the contact, friction, heat and link-candidate passes
against the FP32 oracle: snow sets on either side of each line between the forms, cells of more
than 32 members, contact lists longer than one warp, links formed in the step as well."""
import numpy as np
import pytest

from snowsimulation_b200 import scene
from snowsimulation_b200.abi import QUIRKS_FIXED, QUIRKS_REFERENCE
from tests._util import diff_worlds

pytestmark = pytest.mark.gpu

SCENES = {   # snow sizes: 9,000 | 9,261, 15,984 | 16,016, 23,976 | 24,024 around the lines
    "one": dict(water=(1, 1, 1), snow=(1, 1, 1)),
    "cells of 60": dict(water=(4, 4, 4), snow=(9, 9, 9), spacing=0.0103),
    "contact lists overflow": dict(water=(3, 3, 3), snow=(9, 9, 9), spacing=0.0077),
    "9000": dict(water=(6, 6, 6), snow=(20, 18, 25)),
    "9261": dict(water=(6, 6, 6), snow=(21, 21, 21)),
    "15984": dict(water=(5, 5, 5), snow=(24, 18, 37)),
    "16016": dict(water=(5, 5, 5), snow=(22, 26, 28)),
    "23976": dict(water=(5, 5, 5), snow=(24, 27, 37)),
    "24024": dict(water=(5, 5, 5), snow=(22, 26, 42)),
}


@pytest.mark.parametrize("quirks", [QUIRKS_REFERENCE, QUIRKS_FIXED])
@pytest.mark.parametrize("name", sorted(SCENES))
def test_small_forms_match_oracle(cuda, name, quirks):
    from oracle.oracle import OracleWorld
    from snowsimulation_b200.world import Simulation
    kw = dict(SCENES[name])
    s = kw.pop("spacing", 0.02)
    w = scene.scene_drop(kw.pop("water"), kw.pop("snow"), seed=9, spacing=s, water_jitter=0.1 * s,
                         snow_jitter=0.1 * s, drop_height=0.006, name=name)
    # moving fast enough for a stale list (friction falls back to the traversal) in one step of two
    rng = np.random.default_rng(3)
    w.dem["velocity"][:] = rng.uniform(-1.5, 1.5, w.dem["velocity"].shape).astype(np.float32)
    g = Simulation(w, quirks=quirks)
    o = OracleWorld(w, 32, quirks=quirks)
    g.setup()
    o.setup()
    for _ in range(3):
        g.step()
        o.step()
        assert not diff_worlds(o.w, g.to_host())
