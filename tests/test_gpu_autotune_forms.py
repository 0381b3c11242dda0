"""The tuner keeps the forms of a pass apart: one warp per particle in the buckets from 32 on, one
thread per particle below, each timed by itself; a table tuned on one kind of scene says nothing
about the other kind's kernels, and the steps it shapes keep their results."""
import pytest

from snowsimulation_b200 import autotune, scene
from tests._util import diff_worlds

pytestmark = pytest.mark.gpu
PASSES = ("k_density<false>", "k_density<true>", "k_heat", "k_link_filter", "k_dem_corr<true>", "k_friction<true>")


@pytest.mark.parametrize("snow,warp,thread", [
    ((8, 5, 8), PASSES, ()),                                            # 320 snow: every pass one warp each
    ((24, 18, 24), set(PASSES) - {"k_heat"}, {"k_heat", "k_friction<true>"}),   # 10,368: both friction forms run
    ((40, 34, 40), (), PASSES),                                         # 54,400: one thread each
])
def test_forms_are_tuned_apart(cuda, snow, warp, thread):
    from snowsimulation_b200.world import Simulation

    def make():
        return Simulation(scene.scene_drop((4, 4, 4), snow, seed=7, water_jitter=0.002, snow_jitter=0.002,
                                           drop_height=0.01, init_links=True)).setup()
    autotune.reset()
    ref = make()
    ref.step(substeps=2, use_graph=True)
    sim = make()
    try:
        rows = [line.split() for line in autotune.tune(sim, substeps=1).splitlines()]
        buckets = {p: {int(r[1]) >= 32 for r in rows if r[0] == p} for p in PASSES}
        assert {p for p in PASSES if True in buckets[p]} == set(warp)
        assert {p for p in PASSES if False in buckets[p]} == set(thread)
        assert not any("_warp<" in r[0] or r[0] in ("k_heat_warp", "k_link_filter_warp") for r in rows)
        sim.step(substeps=2, use_graph=True)
        assert not diff_worlds(ref.to_host(), sim.to_host())
    finally:
        autotune.reset()
