"""Link formation against the FP32 oracle at the sizes where a colour pass changes its path:
super-cells with fewer and more active particles than one batch, particles with fewer and
more candidates than the shared-memory list holds, dynamic caps, one snow particle."""
import pytest

from snowsimulation_b200 import scene
from snowsimulation_b200.abi import QUIRKS_FIXED, QUIRKS_REFERENCE

from tests._util import diff_worlds

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("snow,spacing,dynamic,quirks", [
    ((1, 1, 1), 0.02, False, QUIRKS_REFERENCE),
    ((3, 3, 3), 0.02, False, QUIRKS_FIXED),        # fewer candidates than a warp
    ((9, 5, 7), 0.02, False, QUIRKS_REFERENCE),    # 64 particles a super-cell: two batches
    ((8, 8, 8), 0.013, False, QUIRKS_FIXED),       # about 100 candidates: past the shared list
    ((7, 6, 9), 0.016, True, QUIRKS_REFERENCE),    # dynamic caps, about 64 candidates
])
def test_links_match_oracle(cuda, snow, spacing, dynamic, quirks):
    from oracle.oracle import OracleWorld
    from snowsimulation_b200.world import Simulation
    w = scene.scene_drop((2, 2, 2), snow, seed=3, spacing=spacing, snow_jitter=0.1 * spacing, drop_height=0.03,
                         init_links=True, name="links")
    w.flags["dynamic_max_connections"] = dynamic
    g = Simulation(w, quirks=quirks).setup()
    o = OracleWorld(w, 32, quirks=quirks).setup()
    assert not diff_worlds(o.w, g.to_host())
    for _ in range(3):
        g.step()
        o.step()
        assert not diff_worlds(o.w, g.to_host())
