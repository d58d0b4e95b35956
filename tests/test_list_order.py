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


# one cell of n droplets: ranking blocks hold 128 sorted positions
@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 257, 1000])
@pytest.mark.gpu
@pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")
def test_rank_within_a_cell(n):
    import ntlp_b200
    import pyoracle
    case = small_case(n=n + 40, grid_n=(6, 5, 7), params=gen.default_params(icase=0))
    d = clone(case.droplets)
    g = case.grid
    rng = np.random.Generator(np.random.Philox(5))
    one = rng.permutation(n + 40)[:n]                      # the cell's droplets, spread over the list
    for a, (lo, w) in enumerate(((2 * g["xl"] / 6, g["xl"] / 6), (2 * g["yl"] / 5, g["yl"] / 5),
                                 (g["zz"][3], g["zz"][4] - g["zz"][3]))):
        d["xp"][a][one] = lo + w * (0.3 + 0.4 * rng.random(n))
    d["vp"][:, one] = 0.0
    s = ntlp_b200.DropletStep(g, case.params, capacity=n + 40)
    ext = case.ext()
    s.set_fields_ext(ext)
    s.set_droplets(d)
    s.particle_update_BE(1e-4, 2)
    o = pyoracle.Oracle(g, case.params, ext)
    od = clone(d)
    o.step_be(od, 1e-4, 2)
    want, _ = o.coupling(od, 1e-4)                         # sums in list order: the ranks decide the bits
    for q, got in enumerate(s.particle_coupling_update(1e-4)):
        assert np.array_equal(np.asarray(got).view(np.int64), want[q].view(np.int64)), q
    s.close()


# device read-backs of few and of many arrays: direct gathers up to two values,
# records of 4, 8, 12 and 16, and more than one record
@pytest.mark.parametrize("keys", [("Tp",), ("Tp", "radius"), ("xp",), ("xp", "Tp"), ("xp", "vp", "rc"), ("xp", "vp", "uf"),
                                  ("xp", "vp", "uf", "vp_old", "Tp", "Tf", "radius"),
                                  ("xp", "vp", "uf", "vp_old", "Tp", "Tf", "radius", "qinf", "qstar", "mult", "lid")])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.gpu
@pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")
def test_device_read_back_of_any_arrays(keys, precision):
    import ntlp_b200
    case = small_case(n=1500, grid_n=(12, 10, 16), params=gen.default_params(icase=1, precision=precision))
    d = clone(case.droplets)
    d["xp"][2][::5] = 0.1 * d["radius"][::5]               # some die at the floor
    d["vp"][2][::5] = -5.0
    s = ntlp_b200.DropletStep(case.grid, case.params, capacity=1700)
    s.set_fields_ext(case.ext())
    s.set_droplets(d)
    for it in (2, 3):
        s.particle_update_BE(case.dt, it)
        dev = s.get_droplets_device(keys=keys)             # between steps: the next one must not notice
        host = s.get_droplets()
        for k in keys:
            assert np.array_equal(dev[k].cpu().numpy(), host[k]), (it, k)
    s.close()
    t = ntlp_b200.DropletStep(case.grid, case.params, capacity=1700)
    t.set_fields_ext(case.ext())
    t.set_droplets(d)
    for it in (2, 3):
        t.particle_update_BE(case.dt, it)
    for k, v in t.get_droplets().items():
        assert np.array_equal(v, host[k]), k
    t.close()
