"""What a pair of CTAs waits for after an abort (``csrc/pair_drain.cuh``), built for the host: two
loaders that stop anywhere in a ring whose barriers are counted as the hardware counts them, copies
that land in any order.  Every wait of the drain ends, and none of the copies is left under way.
Needs g++ only."""
import os
import shutil
import subprocess

import pytest

from util import ROOT

HARNESS = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "pair_drain.cuh"

struct Barrier {                       // one arrival a phase, and the bytes
    int pending = 1, phase = 0;
    long bytes = 0;
    void settle() { if (pending == 0 && bytes == 0) pending = 1, ++phase; }
    void arrive_expect(long n) { bytes += n; --pending; settle(); }
    void complete(long n) { bytes -= n; settle(); }
};

int main() {
    constexpr long SIZE = 1000;
    srand(7);
    int bad = 0;
    for (int run = 0; run < 20000; ++run) {
        const int stages = 1 + rand() % 8, steps = rand() % 200;
        std::vector<Barrier> full(stages);
        std::vector<int> flying;       // the barrier of each copy (half a CTA's bytes) under way
        auto land = [&] {
            const int at = rand() % (int)flying.size(), s = flying[at];
            flying.erase(flying.begin() + at);
            full[s].complete(SIZE / 2);
        };
        int issued[2] = {0, 0}, consumed = 0;
        const int bias = rand() % 5;
        for (int step = 0; step < steps; ++step) {
            const int what = rand() % 8, cta = rand() % 4 < bias ? 1 : 0;
            if (what < 4) {            // a loader, if its stage is free
                const int i = issued[cta], s = i % stages;
                if (i - consumed >= stages) continue;
                if (cta == 0) full[s].arrive_expect(2 * SIZE);
                flying.push_back(s);
                flying.push_back(s);
                ++issued[cta];
            } else if (what < 7) {
                if (!flying.empty()) land();
            } else if (full[consumed % stages].phase > consumed / stages) {
                ++consumed;            // the products
            }
        }
        pair_drain(issued[0], issued[1], stages,
                   [&](int s) { full[s].arrive_expect(SIZE); },
                   [&](int s) { full[s].complete(SIZE); },
                   [&](int s, int parity) {
                       while ((full[s].phase & 1) == parity && !flying.empty()) land();
                       if ((full[s].phase & 1) == parity) ++bad;      // would run to its limit
                   });
        bad += !flying.empty();
    }
    printf("bad %d\n", bad);
    return bad ? 1 : 0;
}
"""


def test_a_pair_leaves_no_copy_under_way(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    (tmp_path / "pair.cc").write_text(HARNESS)
    subprocess.run([gxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-Wno-unknown-pragmas", "-I",
                    os.path.join(ROOT, "agave_b200", "csrc"), str(tmp_path / "pair.cc"), "-o",
                    str(tmp_path / "pair")], check=True)
    run = subprocess.run([str(tmp_path / "pair")], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, (run.returncode, run.stdout, run.stderr[:2000])
