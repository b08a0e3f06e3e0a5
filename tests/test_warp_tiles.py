"""CPU test of the sizes of warp tiles (tile_ranges): short chains beside long linear
chains, beside branched ones and alone, in plans of many beads, so that their tiles are
as large as they come.  A lane names a tile's bead pairs by the bits of a 32-bit word, a
row of 32 pairs each, so a tile of linear chains has 1,024 pairs at most, a chain of an
odd length one more than half its beads.  The tiles of an architecture are also no
larger than the form's buffer and hold every chain once."""
import os
import subprocess

import new_arch_b200.build as build

PROGRAM = r"""
#include <cstdio>
#include <initializer_list>
#include "scmf_engine.h"
using namespace scmf;
// length 0: combs of 40 (no linear chain)
static int check(std::initializer_list<Plan::Chains> chains, bool screened) {
    Plan p;
    for (Plan::Chains c : chains) {
        c.screen = screened && c.length > 1 ? kScreenAll : kScreenOff;
        p.chains.push_back(c);
        p.linear = p.linear && c.linear;
        p.max_length = c.length > p.max_length ? c.length : p.max_length;
        p.max_deg = c.linear ? 2 : 3;
    }
    int form = -1, bad = 0;
    const auto ranges = tile_ranges(p, &form);
    if (ranges.size() != p.chains.size()) {
        std::printf("%zu ranges of %zu\n", ranges.size(), p.chains.size());
        return 1;
    }
    int first = 0;
    for (size_t i = 0; i < ranges.size(); ++i) {
        const SweepArch& r = ranges[i];
        const int pairs = r.per * ((r.length + 1) / 2), beads = r.per * r.length;
        if (r.per < 1 || beads > kSweepForms[form].beads || r.first != first || r.n_chains != p.chains[i].n_chains ||
            (p.chains[i].linear && pairs > 32 * 32)) {
            std::printf("form %d: %d chains of %d a tile, %d pairs\n", form, r.per, r.length, pairs);
            bad = 1;
        }
        first += (r.n_chains + r.per - 1) / r.per;
    }
    return bad;
}
int main() {
    int bad = 0;
    const auto of = [](int length, long long beads, bool linear) {
        return Plan::Chains{nullptr, nullptr, length, (int)(beads / length), linear, 0, kScreenOff};
    };
    for (int screened = 0; screened < 2; ++screened)
        for (int length = 1; length <= 64; ++length)
            for (long long beads : {100000ll, 1400000ll, 16000000ll, 100000000ll}) {
                const auto c = of(length, beads, true);
                bad |= check({c}, screened);
                bad |= check({of(40, 2000000, false), c}, screened);
                for (int other : {961, 970, 1200, 1900, 1984}) bad |= check({of(other, 1200000, true), c}, screened);
                bad |= check({of(1280, 400000, false), of(1279, 400000, true), c}, screened);
            }
    return bad;
}
"""


def test_tiles_fit_a_lanes_mask(tmp_path):
    lib = build.LIB
    src, exe = tmp_path / "tiles.cpp", tmp_path / "tiles"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", build.INC, "-I", build.CSRC, "-I",
                    os.path.join(build.CUDA, "include"), str(src), "-o", str(exe), "-L", os.path.dirname(lib), "-lscmf",
                    "-Wl,-rpath," + os.path.dirname(lib)], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout[:2000]
