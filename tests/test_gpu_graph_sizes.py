"""A host that adds or removes particles between calls keeps its captured graph: the sizes live on
the device, so only a change of a pass's form captures again.  Captures are counted from the CUDA
runtime's calls, and the replayed steps equal the same steps launched one by one."""
import pytest
import torch

from snowsimulation_b200 import scene
from snowsimulation_b200.abi import QUIRKS_FIXED, QUIRKS_REFERENCE
from tests._util import diff_worlds

pytestmark = pytest.mark.gpu


def _captures(f):
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA], acc_events=True) as p:
        f()
        torch.cuda.synchronize()
    return sum(e.name.startswith("cudaGraphInstantiate") for e in p.events())


@pytest.mark.parametrize("quirks", [QUIRKS_REFERENCE, QUIRKS_FIXED])
def test_sizes_do_not_capture_again(cuda, quirks):
    from snowsimulation_b200.world import Simulation
    a, b = (Simulation(scene.tiny(seed=4, water=(6, 6, 6), snow=(8, 5, 8), init_links=True), quirks=quirks).setup()
            for _ in range(2))

    def shrink(sim, use_graph):
        for _ in range(6):
            sim.n_sph -= 7      # the host takes its last water particles out
            sim.step(use_graph=use_graph)

    assert _captures(lambda: a.step(use_graph=True)) == 1
    assert _captures(lambda: shrink(a, True)) == 0
    b.step()
    shrink(b, False)
    assert not diff_worlds(a.to_host(), b.to_host())
