"""Link formation packs particle indices into 25 bits, as the substep's neighbour lists do: sets of
2^25 particles are refused as the substep refuses them, before anything is allocated or launched."""
import ctypes as C

import pytest

from snowsimulation_b200 import _native
from snowsimulation_b200.abi import Batch, CellData, ParticleDeviceData
from snowsimulation_b200.params import make_sim_params


@pytest.mark.parametrize("batch", [False, True])
def test_connect_refuses_indices_beyond_25_bits(batch):
    lib = _native.load()
    p = make_sim_params()
    assert lib.snowb_set_sim_params(C.byref(p)) == 0
    dem, cells = ParticleDeviceData(), CellData()
    if batch:
        b = Batch(1, 1, 0, 8, 0, 0)     # the ids are not read by a refused call
        rc = lib.snowb_batch_connect_and_record(C.byref(b), C.byref(dem), 1 << 25, cells, 0)
    else:
        rc = lib.snowb_connect_and_record(C.byref(dem), 1 << 25, cells, 0)
    assert rc == -1
    assert b"2^25" in lib.snowb_last_error_string()
