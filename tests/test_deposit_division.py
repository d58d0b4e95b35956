"""The FP64 deposition's division by reciprocal: bit-exact against the oracle
where it applies, and where it has to give way to the division (a denominator
whose significand is all ones, factors below its range)."""
import numpy as np
import pytest

from conftest import cuda_available
from helpers import bitwise_equal, clone
from ntlp_b200 import abi
from ntlp_b200 import generator as gen

ONES = 2.0 - 2.0 ** -52          # significand of all ones


@pytest.mark.parametrize("grid_n,extent,tiny", [
    ((8, 6, 9), (2.0, 2.0, 2.0), False),                  # reciprocals
    ((8, 6, 9), (8 * ONES, 7.0, 3.0), False),             # dx = 2 - 2^-52: divides
    ((8, 6, 9), (2.0, 2.0, 2.0), True),                   # factors of 1e-297: those tiles divide
    ((5, 3, 40), (1.0, 0.3, 4.0), False),                 # ragged: images across narrow boxes
    ((2, 2, 3), (2.0, 2.0, 2.0), False),                  # the smallest grid
])
@pytest.mark.gpu
@pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")
def test_fp64_sources_bit_exact(grid_n, extent, tiny):
    import ntlp_b200
    import pyoracle
    params = gen.default_params(ievap=0 if tiny else 1, icase=0)
    grid = gen.make_grid(*grid_n, *extent)
    fields = gen.make_fields(grid, 3, rms=0.3)
    d = gen.make_droplets(grid, fields, params, 1500, 3)
    if tiny:
        up = d["xp"][2] > 0.5 * extent[2]
        d["radius"][up] = 1e-100
        d["m_s"][up] = 1e-303
    d["mult"] = 1 + np.arange(1500, dtype=np.int64) % 7
    ext = {k: gen.to_ext(grid, v) for k, v in fields.items()}
    s = ntlp_b200.DropletStep(grid, params, capacity=1500)
    s.set_fields_ext(ext)
    s.set_droplets(d)
    o = pyoracle.Oracle(grid, params, ext)
    od = clone(d)
    for it in (2, 3):
        s.particle_update_BE(1e-3, it)
        o.step_be(od, 1e-3, it)
    for layout in (abi.NTLP_LAYOUT_COLUMN,):
        got = s.particle_coupling_update(1e-3, layout=layout)
        want, _ = o.coupling(od, 1e-3)
        for q in range(6):
            assert bitwise_equal(np.asarray(got[q]), want[q]), q
    s.close()


# densities on both sides of each stage capacity of the FP64 tiles, and above all of them
@pytest.mark.parametrize("n", [1300, 1450, 2600, 2900, 9000, 9500, 20000])
@pytest.mark.gpu
@pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")
def test_fp64_stage_capacities(n):
    import ntlp_b200
    import pyoracle
    params = gen.default_params(icase=0)
    grid = gen.make_grid(9, 9, 12, 2.0, 2.0, 2.0)              # 1300 cells
    fields = gen.make_fields(grid, 3, rms=0.3)
    d = gen.make_droplets(grid, fields, params, n, 3)
    ext = {k: gen.to_ext(grid, v) for k, v in fields.items()}
    s = ntlp_b200.DropletStep(grid, params, capacity=n)
    s.set_fields_ext(ext)
    s.set_droplets(d)
    s.particle_update_BE(1e-3, 2)
    o = pyoracle.Oracle(grid, params, ext)
    od = clone(d)
    o.step_be(od, 1e-3, 2)
    want, _ = o.coupling(od, 1e-3)
    for _ in range(2):                                         # the overflow list is empty again
        for q, got in enumerate(s.particle_coupling_update(1e-3)):
            assert bitwise_equal(np.asarray(got), want[q]), q
    s.close()
