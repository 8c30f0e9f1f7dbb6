"""The grouping of a solve's columns by their refinement state, on the host (no GPU): csrc/refine.h
compiled into a small program that reads one line per call."""
import subprocess

import pytest

from conftest import ROOT

CSRC = ROOT / "treams-rs_b200" / "csrc"
PROGRAM = r"""
#include <cstdio>
#include <iostream>
#include <string>
#include "refine.h"
// p target limit, then p norms of right-hand sides, then rows of p residual norms until the end:
// per row whether a sweep follows, then sweeps per group, whether a group needs the fallback
int main() {
    int p; double target, limit;
    std::cin >> p >> target >> limit;
    auto num = [] { std::string s; std::cin >> s; return s.empty() ? -1.0 : std::stod(s); };
    std::vector<double> bn(p), r(p);
    for (double& v : bn) v = num();
    tcu::RefineGroups g(p, target, 10, false);
    for (;;) {
        for (double& v : r) v = num();
        if (!std::cin) break;
        std::printf("%d ", (int)g.advance(r, bn));
    }
    for (auto& q : g.g) std::printf("%d ", q.sweeps);
    std::printf("%d\n", (int)g.any_above(bn, limit));
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("refine")
    (d / "main.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CSRC}", str(d / "main.cpp"), "-o", str(d / "main")], check=True)

    def run(p, bn, rows, target=1e-13, limit=1e-12):
        text = f"{p} {target} {limit}\n" + " ".join(map(str, bn)) + "\n"
        text += "\n".join(" ".join(map(str, r)) for r in rows) + "\n"
        out = subprocess.run([str(d / "main")], input=text, capture_output=True, text=True, check=True).stdout.split()
        return [int(v) for v in out]

    return run


def test_groups_converge_separately(program):
    # nine columns: a group of eight that is done after one sweep, a column that takes two more
    rows = [[1e-14] * 8 + [1e-6], [1e-14] * 8 + [1e-10], [1e-14] * 8 + [1e-15]]
    assert program(9, [1.0] * 9, rows) == [1, 1, 0, 1, 3, 0]


@pytest.mark.parametrize("column", [0, 3, 8])
@pytest.mark.parametrize("bad", ["nan", "inf"])
def test_a_residual_that_is_no_number_stops_and_falls_back(program, column, bad):
    row = [1e-14] * 9
    row[column] = bad
    assert program(9, [1.0] * 9, [row]) == [0, 1, 1, 1]
    # also when it comes from a correction, and beside columns that still converge
    rows = [[1e-6] * 9, [1e-9] * 9]
    rows[1][column] = bad
    assert program(9, [1.0] * 9, rows)[-1] == 1


def test_a_right_hand_side_that_is_no_number_does_not_fall_back(program):
    assert program(2, ["nan", 1.0], [["nan", 1e-14]]) == [0, 1, 0]
