"""The FP64 deposition's stage capacity, chosen per box from the droplets it was
given: the rule and the order of a batch's tiles on the CPU, and on the GPU
contexts with much room to spare and batches of boxes of different densities
against each box alone, eager and as a graph, with new droplets in between."""
import subprocess

import numpy as np
import pytest

from conftest import ROOT, cuda_available
from helpers import STATE_KEYS, bitwise_equal
from ntlp_b200 import abi
from ntlp_b200 import generator as gen

PROGRAM = r"""
#include <cstdio>
#include "ntlp_stage64.h"
using namespace ntlp;
int main() {
    int bad = 0;
    // droplets per tile on both sides of each line (m + 4 sqrt(m) = 640 at m = 546.5, 3840 at 3600)
    const struct { long long n; int cap; } at[] = {{0, 0}, {546, 0}, {547, 1}, {1300, 1}, {1301, 2}, {3599, 2},
                                                   {3601, 0}, {100000, 0}};
    for (int cells : {425, 495, 585})
        for (auto &a : at) bad += deposit64_cap(a.n * 1000, 1000LL * cells, cells) != a.cap;
    // every box once, in runs that cover the table, at most two, each box in a run that stages enough
    for (int m = 0; m < 81; ++m) {
        std::vector<int> cap, tiles, order;
        std::vector<TileRun> runs;
        for (int k = 0, r = m; k < 4; ++k, r /= 3) { cap.push_back(r % 3); tiles.push_back(5 + 7 * k); }
        deposit64_order(cap, tiles, order, runs);
        bad += order.size() != 4 || runs.empty() || runs.size() > 2;
        int at = 0, box = 0, seen = 0;
        for (auto &r : runs) {
            bad += r.first != at;
            for (int left = r.count; left > 0; ++box) {
                left -= tiles[order[box]];
                bad += left < 0 || cap[order[box]] > r.cap || (cap[order[box]] == 2) != (r.cap == 2);
                seen |= 1 << order[box];
            }
            at += r.count;
        }
        bad += seen != 15 || at != 5 + 12 + 19 + 26;
    }
    printf("%d\n", bad);
    return 0;
}
"""


def test_rule_and_order(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=address,undefined", "-I", f"{ROOT}/ntlp_b200/csrc",
                    str(src), "-o", str(exe)], check=True, timeout=300)
    r = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60)
    assert r.stdout.strip() == "0", r.stdout


GRIDS = [(9, 9, 12), (8, 6, 15), (12, 5, 9), (4, 7, 33)]


def _case(b, density):
    grid = gen.make_grid(*GRIDS[b], 2.0, 2.0, 2.0)
    params = gen.default_params(icase=0, precision=abi.NTLP_PREC_FP64)
    fields = gen.make_fields(grid, 3 + b, rms=0.3)
    n = int(density * (grid["nnx"] + 1) * (grid["nny"] + 1) * (grid["nnz"] + 1))
    d = gen.make_droplets(grid, fields, params, n, 5 + b)
    return grid, params, {k: gen.to_ext(grid, v) for k, v in fields.items()}, d


def _launches(s):
    s.profile_read()
    s.particle_coupling_update(1e-3, download=False)
    return s.profile_read()["launches"]


def _alone(case, room):
    import ntlp_b200
    grid, params, ext, d = case
    s = ntlp_b200.DropletBatch([grid], params, [room])
    s.set_box_fields_ext(0, ext)
    s.set_box_droplets(0, d)
    return s


# densities per box; launches of one deposition (its runs, the overflow tiles, the fold)
@pytest.mark.parametrize("first,then", [
    ((0.5, 4.0, 1.6, 5.0), (4.0, 0.5, 0.5, 9.0)),     # two runs, interleaved; then others
    ((0.5, 0.7, 1.0, 0.1), (0.5, 4.0, 1.0, 0.1)),     # one run; then two
    ((4.0, 5.0, 4.5, 5.5), (9.0, 9.0, 9.0, 9.0)),     # one run of the largest stage; then none that stages
])
@pytest.mark.gpu
@pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")
def test_batch_of_uneven_boxes(first, then):
    import ntlp_b200
    cases = [[_case(b, d) for b, d in enumerate(dens)] for dens in (first, then)]
    params = cases[0][0][1]
    room = [max(c[3]["radius"].shape[0] for c in pair) for pair in zip(*cases)]
    a = ntlp_b200.DropletBatch([c[0] for c in cases[0]], params, room)
    for dens, part in zip((first, then), cases):
        for b, c in enumerate(part):
            a.set_box_fields_ext(b, c[2])
            a.set_box_droplets(b, c[3])
        big = [2.7 < x < 6.0 for x in dens]                 # boxes of the largest stage, whatever the tile shape
        a.particle_update_BE(1e-3, 1)
        assert _launches(a) == len(set(big)) + 2
        a.advance_graph(1e-3, 2, 2)
        a.sync()
        for b, c in enumerate(part):
            s = _alone(c, room[b])
            for it in (1, 2, 3):
                s.particle_update_BE(1e-3, it)
                s.particle_coupling_update(1e-3, download=False)
            got, want = a.get_box_droplets(b), s.get_box_droplets(0)
            for k in STATE_KEYS:
                assert bitwise_equal(got[k], want[k]), (b, k)
            for q, (x, y) in enumerate(zip(a.box_sources(b), s.box_sources(0))):
                assert bitwise_equal(np.asarray(x), np.asarray(y)), (b, q)
            s.close()
    a.close()


@pytest.mark.parametrize("density", [0.5, 1.6, 4.0])
@pytest.mark.gpu
@pytest.mark.skipif(not cuda_available(), reason="needs a CUDA device")
def test_room_to_spare(density):
    """The room for droplets changes neither the results nor the launches."""
    c = _case(0, density)
    n = c[3]["radius"].shape[0]
    out = []
    for room in (n, 3 * n, 8 * n):
        s = _alone(c, room)
        s.particle_update_BE(1e-3, 1)
        assert _launches(s) == 3
        out.append([np.asarray(x).copy() for x in s.box_sources(0)])
        s.close()
    for o in out[1:]:
        for q in range(6):
            assert bitwise_equal(out[0][q], o[q]), q
