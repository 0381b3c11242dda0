"""The reverse passes in their one-thread form against the one-warp form: a small scene alone, and the
same scene beside a block of snow that is out of its reach and brings the sets past the line
between the forms.  The small scene's part of the gradient is the same, bit for bit; the parameter
gradients, which all particles' (zero) parts join in another order, to float32 rounding."""
import numpy as np
import pytest
import torch

from snowsimulation_b200 import adjoint, scene
from snowsimulation_b200.abi import QUIRKS_FIXED

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [{}, {"dem_friction": False}, {"compute_temperature": False, "dem_viscosity": False}])
def test_one_thread_form_equals_one_warp_form(cuda, flags):
    from snowsimulation_b200.world import Simulation
    g = np.random.default_rng(5)
    water = scene.lattice((6, 5, 6), 0.02, (-0.75, 0.075, -0.05), 0.002, g)
    near = scene.lattice((8, 4, 8), 0.02, (-0.77, 0.01, -0.07), 0.002, g)
    far = scene.lattice((50, 30, 50), 0.02, (-0.09, 0.01, -0.49), 0.002, g)
    out = []
    for snow in (near, np.concatenate([near, far])):
        w = scene.build_world(water, snow, 100.0, -10.0, init_links=True)
        w.flags["change_phase"] = False
        w.flags.update(flags)
        sim = Simulation(w, quirks=QUIRKS_FIXED).setup()
        n = len(near)
        v = sim.sph.t["velocity"][:sim.n_sph].clone().requires_grad_(True)
        th = adjoint.params_of(sim).requires_grad_(True)
        xs, xd, Ts, Td = adjoint.rollout(sim, v, th, 4, 2)
        ((xd[:n].double() ** 2).sum() + (xs.double() ** 2).sum() + 1e-4 * (Td[:n].double() ** 2).sum()
         + 1e-4 * (Ts.double() ** 2).sum()).backward()
        out.append((xs.detach(), xd[:n].detach(), Ts.detach(), Td[:n].detach(), v.grad, th.grad))
    a, b = out
    for x, y in zip(a[:5], b[:5]):
        assert torch.equal(x, y)
    assert float(a[4].abs().max()) > 0
    assert torch.allclose(a[5], b[5], rtol=1e-4, atol=0)
