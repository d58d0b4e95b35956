"""The FP64 deposition's division by reciprocal: bit-exact against the oracle
where it applies, and where it has to give way to the division (a denominator
whose significand is all ones, factors below its range)."""
import subprocess

import numpy as np
import pytest

from conftest import ROOT, cuda_available
from helpers import bitwise_equal, clone
from ntlp_b200 import abi
from ntlp_b200 import generator as gen

ONES = 2.0 - 2.0 ** -52          # significand of all ones


PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <vector>
#include "ntlp_recip.h"
using namespace ntlp;
int main() {
    int bad = 0;
    const int nnz = 5, n = nnz + 3;
    std::vector<double> rec(2 * n);
    auto use = [&](double dx, double dy, std::vector<double> dzu) {
        return deposit_reciprocals(dx, dy, dzu.data(), nnz, rec.data());
    };
    const double ones = 2.0 - 0x1p-52, unset[] = {0.25, 0.0, -1.0, 1e-300, INFINITY, NAN, ones};
    for (double u : unset)                                  // the levels that no cell has
        for (double w : unset) {
            bad += !use(0.5, 0.75, {u, 0.1, 0.2, 0.3, 0.4, 0.5, 0.6, w});
            const double dz[] = {0, 0.1, 0.2, 0.3, 0.4, 0.5, 0.6};
            for (int k = 1; k <= nnz + 1; ++k)
                bad += rec[k] != 1.0 / dz[k] || rec[n + k] != 1.0 / (0.5 * 0.75 * dz[k]);
            for (int k : {0, nnz + 2}) bad += rec[k] != 1.0 || rec[n + k] != 1.0;
        }
    for (int k = 1; k <= nnz + 1; ++k)                      // those that one has
        for (double u : unset) {
            std::vector<double> dzu = {1, 0.1, 0.2, 0.3, 0.4, 0.5, 0.6, 1};
            dzu[k] = u;
            bad += use(0.5, 0.75, dzu) != (u == 0.25);
        }
    bad += use(ones, 1, {1, 1, 1, 1, 1, 1, 1, 1}) || use(1, ones, {1, 1, 1, 1, 1, 1, 1, 1});
    printf("%d\n", bad);
    return 0;
}
"""


def test_which_grids_divide_by_reciprocal(tmp_path):
    """Every level of a cell has to qualify; dzu(0) and dzu(nnz+2), which callers may
    leave unset, do not count."""
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-fsanitize=address,undefined",
                    "-fno-sanitize=float-divide-by-zero", "-I", f"{ROOT}/ntlp_b200/csrc", str(src), "-o", str(exe)],
                   check=True, timeout=300)
    r = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60)
    assert r.stdout.strip() == "0", r.stdout


@pytest.mark.parametrize("grid_n,extent,tiny", [
    ((8, 6, 9), (2.0, 2.0, 2.0), False),                  # reciprocals
    ((8, 6, 9), (8 * ONES, 7.0, 3.0), False),             # dx = 2 - 2^-52: divides
    ((8, 6, 9), (2.0, 2.0, 2.0), True),                   # factors of 1e-297: those tiles divide
    ((5, 3, 40), (1.0, 0.3, 4.0), False),                 # ragged: images across narrow boxes
    ((2, 2, 3), (2.0, 2.0, 2.0), False),                  # the smallest grid
    ((8, 6, 10), (2.0, 2.0, 2.0), False),                 # dzu(0), dzu(nnz+2) left at zero
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
    if grid_n[2] == 10:
        grid["dzu"][[0, -1]] = 0.0
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
