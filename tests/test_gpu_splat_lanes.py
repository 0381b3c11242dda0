"""Point views on either side of the point size up to which one lane takes a sprite (8), bit for bit
against the CPU restatement: sprites of less than a pixel, of a few and of many."""
import numpy as np
import pytest

from snowsimulation_b200 import render, scene
from snowsimulation_b200.export import SNOW_RGB, WATER_RGB

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [8.0, float(np.nextafter(np.float32(8.0), np.float32(9.0)))])
@pytest.mark.parametrize("distance", [0.3, 1.5, 20.0])
def test_both_forms_match_the_restatement(cuda, size, distance):
    from oracle import render_oracle
    from snowsimulation_b200.world import Simulation
    sim = Simulation(scene.scene_drop((5, 5, 5), (9, 7, 9), seed=4, snow_jitter=0.002, water_jitter=0.002)).setup()
    cam = render.camera(eye=(0.1 * distance, 0.1 + 0.3 * distance, distance), center=(0.0, 0.1, 0.0), width=149, height=97,
                        point_size=size)
    got = render.render(sim, cam).cpu().numpy()
    host = sim.to_host()
    ref = render_oracle.render(render.camera_dict(cam), [(host.sph["positions"][:sim.n_sph], None, {"rgb": WATER_RGB}),
                                                         (host.dem["positions"][:sim.n_dem], None, {"rgb": SNOW_RGB})])
    assert (ref[..., 3] > 0).any()
    assert np.array_equal(got, ref, equal_nan=True)
