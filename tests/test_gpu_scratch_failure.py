"""Scratch that does not fit the GPU: the call reports it, and the calls after it work.  The interlink
slots of 2^30 per particle ask for terabytes, which the allocator refuses at once."""
import ctypes as C

import pytest

from snowsimulation_b200 import _native, scene
from snowsimulation_b200.params import make_sim_params
from tests._util import diff_worlds

pytestmark = pytest.mark.gpu


def test_calls_after_a_failed_allocation(cuda):
    from snowsimulation_b200.world import Simulation
    a = Simulation(scene.tiny(seed=5, init_links=True)).setup()
    for _ in range(3):
        a.step()
    b = Simulation(scene.tiny(seed=5, init_links=True)).setup()
    p = make_sim_params()
    p.maximum_connection = 1 << 30
    _native.check(b.lib.snowb_set_sim_params(C.byref(p)))
    rc = b.lib.snowb_connect_and_record(C.byref(b._s[1]), b.n_dem, b._c[1], 0)
    assert rc == -2 and b"cudaMalloc" in b.lib.snowb_last_error_string()
    _native.check(b.lib.snowb_set_sim_params(C.byref(b.params)))
    for _ in range(3):
        b.step()
    assert not diff_worlds(a.to_host(), b.to_host())
