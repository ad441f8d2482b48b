"""The split of a batch between teams of blocks and single blocks: its slots stay below the memory it is
given, and a batch that fits without teams is planned without them where they do not.  Host code,
compiled on its own."""
import shutil
import subprocess

import pytest

from copsandrobbers_gb300 import build as B

PROGRAM = r"""
#include "crgpu_batch_plan.h"
#include <cmath>
#include <cstdio>
#include <cstdlib>
using namespace crgpu;
// argv: blocks, memory in slots of the largest graph, then the vertex counts in descending order
int main(int argc, char** argv) {
    const int blocks = atoi(argv[1]);
    std::vector<double> cost;
    for (int i = 3; i < argc; ++i) cost.push_back(std::pow(atof(argv[i]), 4) / 6);
    const int count = (int)cost.size();
    auto slot = [&](int i) { return i < count ? (size_t)(8 * cost[i]) : (size_t)1; };
    const size_t memory = (size_t)(atof(argv[2]) * slot(0));
    const TeamPlan p = plan_teams(cost, blocks, slot(0), memory, [&](int size) { return blocks / size; }, slot);
    printf("%d %d %d %d %.6f", p.size, p.resident(count), p.count, (int)(p.bytes(count) < memory),
           (double)p.bytes(count) / slot(0));
}
"""


@pytest.fixture(scope="module")
def planner(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("g++ absent")
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", B.CSRC, str(d / "plan.cpp"), "-o", str(d / "plan")], check=True)

    def run(blocks, memory, sizes):
        args = [str(d / "plan"), str(blocks), str(memory), *map(str, sorted(sizes, reverse=True))]
        out = subprocess.run(args, capture_output=True, text=True, check=True).stdout.split()
        return dict(size=int(out[0]), teams=int(out[1]), count=int(out[2]), fits=out[3] == "1", slots=float(out[4]))

    return run


@pytest.mark.parametrize("sizes", [[128] * 10 + [126] * 112, [128 - i // 26 for i in range(126)],
                                   [128] * 3 + [100] * 40, [128] * 16, [96] * 40 + [8] * 100])
def test_plan_stays_within_the_memory(planner, sizes):
    blocks = 152
    teams = planner(blocks, 1e9, sizes)
    assert teams["size"] > 1 and teams["count"] > 0     # such a batch wants teams
    alone = min(len(sizes), blocks)                      # slots of the plan without them
    for memory in (alone * 1.01, alone * 1.5, alone * 2.5, alone * 4.5, alone * 9):
        p = planner(blocks, memory, sizes)
        assert p["fits"], (memory, p)
        assert p["slots"] == pytest.approx(alone) if p["size"] == 1 else p["count"] > 0
    assert planner(blocks, teams["slots"] * 1.01, sizes)["size"] > 1
