"""How zl_advance splits a call between its graphs: a new context's short calls capture no long graph, short
calls keep the graph of two steps beside it where a step is several launches, nothing is left out, and a run of
calls captures a bounded number of graphs."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "graph_plan.h"
// arguments: single_level one_launch nodes calls...; prints per call: run runs pairs direct captured
int main(int argc, char** argv) {
    const bool single = std::atoi(argv[1]), one = std::atoi(argv[2]);
    const long long nodes = std::atoll(argv[3]);
    long long seen = 0;
    int have = 0;
    for (int i = 4; i < argc; ++i) {
        const int steps = std::atoi(argv[i]);
        const zl::GraphPlan p = zl::plan_graph(steps, single, one, nodes, seen, have);
        seen += steps;
        const bool captured = p.runs > 0 && p.run != have;
        if (p.runs > 0) have = p.run;
        std::printf("%d %d %d %d %d\n", p.run, p.runs, p.pairs, p.direct, captured);
    }
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "zllbm_b200", "csrc"), str(d / "plan.cpp"), "-o",
                    str(d / "plan")], check=True)

    def run(single, one, calls, nodes=30000):
        out = subprocess.run([str(d / "plan"), str(int(single)), str(int(one)), str(nodes), *map(str, calls)], capture_output=True,
                             text=True, check=True).stdout
        rows = [tuple(map(int, line.split())) for line in out.splitlines()]
        for steps, (length, runs, pairs, direct, captured) in zip(calls, rows):
            assert runs * length + 2 * pairs + direct == steps and length % 2 == 0
        return rows

    return run


@pytest.mark.parametrize("one", [True, False])
def test_a_new_context_does_not_pay_for_a_long_graph(plan, one):
    for k in (2, 8, 16, 40, 126):
        assert plan(True, one, [k]) == [(0, 0, 0, k, 0) if one else (0, 0, k // 2, 0, 0)]
    assert plan(True, one, [1000])[0][:2] == (16, 62)


def test_short_calls_beside_the_long_graph(plan):
    rows = plan(True, False, [300, 2, 7, 15, 31])
    assert rows == [(16, 18, 6, 0, 1), (16, 0, 1, 0, 0), (16, 0, 3, 1, 0), (16, 0, 7, 1, 0), (16, 1, 7, 1, 0)]
    rows = plan(True, True, [300, 2, 7, 31])
    assert rows == [(16, 18, 0, 12, 1), (16, 0, 0, 2, 0), (16, 0, 0, 7, 0), (16, 1, 0, 15, 0)]


def test_a_program_of_short_calls_gets_a_graph_of_their_length(plan):
    rows = plan(True, True, [8] * 40)
    assert [r[4] for r in rows].index(1) == 15 and rows[-1] == (8, 1, 0, 0, 0)  # the 128th step is in the 16th call
    assert sum(r[4] for r in plan(True, False, list(range(1, 60)) * 3)) <= 5


def test_multi_level_steps_replay_in_pairs(plan):
    assert plan(False, False, [3, 300, 2]) == [(0, 0, 1, 1, 0), (0, 0, 150, 0, 0), (0, 0, 1, 0, 0)]


def test_long_steps_of_one_launch_take_no_graph(plan):
    assert plan(True, True, [1000, 3], 1 << 24) == [(0, 0, 0, 1000, 0), (0, 0, 0, 3, 0)]
    assert plan(True, True, [1000], 1 << 22)[0][:2] == (16, 62)
    assert plan(True, False, [1000], 1 << 24)[0][:2] == (16, 62)
