"""The droplet state read back in list order: every array through the slot
table, with and without killed droplets, to host and to device memory."""
import numpy as np
import pytest

from conftest import cuda_available
from helpers import clone, small_case
from ntlp_b200 import generator as gen


# the tiles of the ranking scan hold 1024 lids, its middle pass 1024 tiles
@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, 5000, 1_050_000])
@pytest.mark.parametrize("killed", [False, True])
@pytest.mark.gpu
@pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")
def test_list_order_and_ranks(n, killed):
    import ntlp_b200
    case = small_case(n=n, grid_n=(12, 10, 16), params=gen.default_params(icase=1))
    d = clone(case.droplets)
    d["xp"][2][:] = 0.5 * case.grid["zl"]
    die = np.zeros(n, dtype=bool)
    if killed:
        die[::3] = True
        if n == 1:
            die[0] = False
        d["xp"][2][die] = 0.1 * d["radius"][die]
        d["vp"][2][die] = -5.0
    d["m_s"] = d["m_s"] * (1.0 + 1e-9 * np.arange(n))       # carried through unchanged
    d["mult"] = np.arange(n, dtype=np.int64) + 1
    s = ntlp_b200.DropletStep(case.grid, case.params, capacity=n)
    s.set_fields_ext(case.ext())
    s.set_droplets(d)
    s.particle_update_BE(case.dt, 2)
    left = np.flatnonzero(~die)
    host = s.get_droplets()
    assert np.array_equal(host["lid"], left)
    assert np.array_equal(host["m_s"], d["m_s"][left])
    assert np.array_equal(host["mult"], d["mult"][left])
    dev = s.get_droplets_device(keys=("xp", "radius", "m_s", "mult", "lid"))
    for k, v in dev.items():
        assert np.array_equal(v.cpu().numpy(), host[k]), k
    s.close()
