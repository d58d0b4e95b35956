"""particle_xy_stats at the edges of its tiles: 64 columns a block, 32 levels a
warp, columns with many and with no droplets."""
import numpy as np
import pytest

from conftest import cuda_available
from helpers import small_case
from ntlp_b200 import generator as gen
from test_stats import _abs_terms, _compare_stats, _oracle


@pytest.mark.parametrize("grid_n,n", [((2, 2, 3), 1), ((7, 7, 31), 900), ((7, 8, 32), 900), ((8, 8, 33), 5000),
                                      ((3, 2, 70), 3000)])
@pytest.mark.gpu
@pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")
def test_stats_at_tile_edges(grid_n, n):
    import ntlp_b200
    case = small_case(n=n, grid_n=grid_n, params=gen.default_params(icase=0))
    case.droplets["xp"][2][: n // 2] *= 0.02               # half of them in the lowest levels
    s = ntlp_b200.DropletStep(case.grid, case.params, capacity=n)
    s.set_fields_ext(case.ext())
    s.set_droplets(case.droplets)
    s.particle_update_BE(case.dt, 1)
    gd = s.get_droplets()
    o = _oracle(case)
    _compare_stats(s.particle_xy_stats(), o.stats(gd), _abs_terms(o, gd))
    assert np.array_equal(s.radius_histogram(), o.radius_histogram(gd))
    s.close()
