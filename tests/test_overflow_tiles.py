"""Mixed deposition tiles above their stage's capacity (768 droplets), which the
overflow kernel merges from global memory, against the per-cell sums that boxes of
large capacity use.  The sources are the same bits."""
import numpy as np
import pytest

from conftest import cuda_available
from helpers import bitwise_equal, small_case
from ntlp_b200 import abi
from ntlp_b200 import generator as gen


@pytest.mark.parametrize("grid_n,n", [
    ((9, 9, 70), 30_000),     # 4.2 a cell: ragged tiles in every direction, above the stage and below
    ((5, 3, 40), 9_000),      # 9 a cell
    ((4, 5, 33), 14_000),     # 14 a cell
    ((2, 2, 3), 2_500),       # 69 a cell, the smallest grid
])
@pytest.mark.gpu
@pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")
def test_overflow_tiles_match_cell_sums(grid_n, n):
    import ntlp_b200
    params = dict(gen.default_params(icase=0), precision=abi.NTLP_PREC_MIXED)
    case = small_case(params=params, n=n, grid_n=grid_n)
    ncells = (grid_n[0] + 1) * (grid_n[1] + 1) * (grid_n[2] + 1)
    out = []
    for cap in (n, max(n, 16 * ncells)):
        s = ntlp_b200.DropletStep(case.grid, params, capacity=cap)
        s.set_fields_ext(case.ext())
        s.set_droplets(case.droplets)
        s.particle_update_BE(case.dt, 1)
        out.append([np.asarray(x).copy() for x in s.particle_coupling_update(case.dt)])
        s.close()
    for q in range(6):
        assert bitwise_equal(out[0][q], out[1][q]), q


@pytest.mark.parametrize("grid_n", [(2, 7, 5), (7, 2, 5), (2, 3, 4), (3, 2, 4), (90, 3, 60), (3, 90, 60)])
@pytest.mark.gpu
@pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")
def test_fold_of_thin_boxes(grid_n):
    """Boxes whose border nodes are all or most of them, and more than one round of
    the fold's blocks: the images folded by a kernel of its own against the folded
    cell sums.  The sources are the same bits."""
    test_overflow_tiles_match_cell_sums(grid_n, 3_000)
