"""The library's buffers are cleared before its first kernels read them, also when the caller's
stream does not wait for the legacy stream and that one is busy."""
import pytest
import torch

from snowsimulation_b200 import _native, scene
from tests._util import diff_worlds

pytestmark = pytest.mark.gpu


def test_new_scratch_beside_a_busy_legacy_stream(cuda):
    from snowsimulation_b200.world import Simulation
    a = Simulation(scene.tiny(seed=6, init_links=True)).setup()
    for _ in range(2):
        a.step()
    a = a.to_host()
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        b = Simulation(scene.tiny(seed=6, init_links=True))
        _native.check(b.lib.snowb_release())
        torch.cuda.synchronize()
        with torch.cuda.stream(torch.cuda.default_stream()):
            torch.cuda._sleep(400_000_000)      # about 0.2 s
        b.setup()
        for _ in range(2):
            b.step()
        assert not diff_worlds(a, b.to_host())
    _native.check(_native.load().snowb_set_stream(None))
