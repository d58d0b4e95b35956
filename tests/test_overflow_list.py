"""The list of deposition tiles left to the overflow kernel, when a deposition is
launched only in part: its tiled kernel ran, the launch of what follows was
refused.  The kernels' own list functions and the host's state, on the CPU,
with a refused launch and a refused clearing: the next deposition lists every
tile once and nothing is written or read past the list."""
import subprocess
import sys

from conftest import ROOT

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "ntlp_overflow.h"
using namespace ntlp;
static int add(int *n) { return (*n)++; }
int main() {
    const int ntiles = 5, guard = -77;
    std::vector<int> mem(2 + ntiles + 64, guard);
    int *list = mem.data();
    list[0] = 0;
    OverflowState s;
    int bad = 0, cleared = 0;
    auto clear = [&] { list[0] = 0; ++cleared; return 0; };
    auto refuse = [&] { return 2; };
    // tiled kernel, overflow kernel, clearing; from `launches` on they are refused
    auto deposit = [&](int launches) {
        std::vector<int> seen(ntiles, 0);
        s.begin();
        if (launches > 0)
            for (int t = 0; t < ntiles; ++t) overflow_put(list, ntiles, t, add);
        if (launches > 1)
            for (int e = 0, n = overflow_count(list, ntiles); e < n; ++e) ++seen[list[1 + e]];
        if (launches > 2) list[0] = 0;
        if (launches < 3) return;
        s.end();
        for (int t = 0; t < ntiles; ++t) bad += seen[t] != 1;
    };
    auto guards = [&] { for (size_t k = 2 + ntiles; k < mem.size(); ++k) bad += mem[k] != guard; };
    bad += s.ready(clear) != 0; deposit(3);
    for (int at = 0; at < 3; ++at) {
        bad += s.ready(clear) != 0; deposit(at); guards();
        bad += s.ready(refuse) != 2;                   // the clearing is refused: reported, asked for again
        bad += s.ready(clear) != 0; deposit(3); guards();
    }
    bad += s.ready(refuse) != 0;                       // nothing to clear after a whole one
    bad += cleared != 3;
    // even without the clearing nothing leaves the list
    deposit(1); deposit(1); deposit(1); guards();
    bad += overflow_count(list, ntiles) != ntiles;
    list[0] = -3;
    bad += overflow_count(list, ntiles) != 0;
    overflow_put(list, ntiles, 1, add); guards();
    printf("%d\n", bad);
    return 0;
}
"""


def test_deposition_launched_in_part(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=address,undefined", "-I", f"{ROOT}/ntlp_b200/csrc",
                    str(src), "-o", str(exe)], check=True, timeout=300)
    r = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60)
    assert r.stdout.strip() == "0", (sys.platform, r.stdout)
