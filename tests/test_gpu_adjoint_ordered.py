"""The reverse pass's ordered warp sums: gradients repeat bit for bit and do not depend on the
checkpoint interval, for particles with fewer neighbours than a warp, with several chunks of
them, and in cells of more than 32 entries with more neighbours than the shared list holds
(their values are checked against the FP64 oracle in test_gpu_adjoint.py)."""
import numpy as np
import pytest

from snowsimulation_b200 import adjoint, scene
from snowsimulation_b200.abi import QUIRKS_FIXED

pytestmark = pytest.mark.gpu


def _scene(spacing, water, snow):
    w = scene.scene_drop(water, snow, seed=9, spacing=spacing, water_jitter=0.1 * spacing, snow_jitter=0.1 * spacing,
                         drop_height=0.6 * spacing, init_links=True, name="adjoint ordered")
    w.flags["change_phase"] = False
    return w


def _grads(w, substeps=2, every=1):
    from snowsimulation_b200.world import Simulation
    sim = Simulation(w, quirks=QUIRKS_FIXED).setup()
    v0 = sim.sph.t["velocity"][:sim.n_sph].clone().requires_grad_(True)
    th = adjoint.params_of(sim).requires_grad_(True)
    target = sim.dem.t["positions"][:sim.n_dem] + 0.003
    _, xd, _, Td = adjoint.rollout(sim, v0, th, substeps, every)
    adjoint.loss_fn(xd, Td, target, Td.detach() + 1.0, 1e-4).backward()
    return v0.grad.cpu().numpy(), th.grad.cpu().numpy()


@pytest.mark.parametrize("spacing,water,snow", [(0.02, (2, 2, 2), (4, 2, 4)),      # fewer neighbours than a warp
                                                (0.012, (4, 3, 4), (7, 5, 7)),    # several chunks
                                                (0.0085, (5, 4, 5), (8, 8, 8))])   # cells past 32, lists past 96
def test_gradients_repeat_and_checkpoints_agree(cuda, spacing, water, snow):
    a, b = _grads(_scene(spacing, water, snow)), _grads(_scene(spacing, water, snow), every=2)
    assert np.isfinite(a[0]).all() and np.isfinite(a[1]).all() and np.abs(a[0]).max() > 0
    assert np.array_equal(a[0], b[0])
    # the scalars are summed with double atomics over at most 1e4 warps: 1e4 * 2^-53 relative
    assert np.allclose(a[1], b[1], rtol=1e4 * 2.0 ** -53, atol=0.0)
