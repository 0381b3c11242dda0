"""Link formation and the substep against the FP32 oracle for other numbers of interlink slots than
the reference's 25: one, a warp's width, and the more than 32 that one thread per super-cell takes."""
import pytest

from snowsimulation_b200 import scene
from snowsimulation_b200.abi import QUIRKS_FIXED, QUIRKS_REFERENCE
from snowsimulation_b200.params import make_sim_params
from tests._util import diff_worlds

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dynamic,quirks", [(False, QUIRKS_REFERENCE), (True, QUIRKS_FIXED)])
@pytest.mark.parametrize("slots", [1, 32, 33, 48])
def test_links_of_other_slot_counts_match_oracle(cuda, slots, dynamic, quirks):
    from oracle.oracle import OracleWorld
    from snowsimulation_b200.world import Simulation
    s = 0.016                                       # about 64 candidates a particle
    w = scene.scene_drop((3, 2, 3), (8, 7, 9), seed=3, spacing=s, snow_jitter=0.1 * s, drop_height=0.02, init_links=True,
                         params=make_sim_params(maximum_connection=slots), name="slots")
    w.flags["dynamic_max_connections"] = dynamic
    g = Simulation(w, quirks=quirks).setup()
    o = OracleWorld(w, 32, quirks=quirks).setup()
    assert not diff_worlds(o.w, g.to_host())
    for _ in range(3):
        g.step()
        o.step()
        assert not diff_worlds(o.w, g.to_host())
