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
PACKED = r"""
#include <cstdio>
#include <iostream>
#include <string>
#include "refine.h"
// p, then rows of residual norms of all columns (target 1e-13): the norms of the packed columns are taken from
// the row by their column, and columns ("x") and norms follow compact()'s moves; per row the packed columns
int main() {
    int p;
    std::cin >> p;
    auto num = [] { std::string s; std::cin >> s; return s.empty() ? -1.0 : std::stod(s); };
    std::vector<double> bn(p, 1.0), row(p), rn(p), packed(p);
    std::vector<int> x(p), out(p, -1);
    for (int c = 0; c < p; ++c) x[c] = c;
    tcu::RefineGroups g(p, 1e-13, 10, false);
    for (;;) {
        for (double& v : row) v = num();
        if (!std::cin) break;
        const int cols = g.columns();
        std::printf("%d ", cols);
        for (int c = 0; c < cols; ++c) packed[c] = row[x[c]];
        g.scatter(packed, rn);
        for (int c = 0; c < cols; ++c)
            if (rn[x[c]] != row[x[c]]) std::printf("norm of %d ", x[c]);
        g.advance(rn, bn);
        g.compact([&](size_t q, int from) { for (int c = 0; c < g.width(q); ++c) out[g.first(q) + c] = x[from + c]; },
                  [&](int from, int to, int width) {
                      if (to + width > from) std::printf("overlap ");
                      for (int c = 0; c < width; ++c) x[to + c] = x[from + c];
                  });
    }
    std::printf("%d\n", g.columns());
    for (int c = 0; c < p; ++c) std::printf("%d ", out[c]);
}
"""


def build(source, d):
    (d / "main.cpp").write_text(source)
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CSRC}", str(d / "main.cpp"), "-o", str(d / "main")], check=True)


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("refine")
    build(PROGRAM, d)

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


@pytest.mark.parametrize("p,slow", [(128, [3]), (128, [0, 7, 15]), (20, [2]), (20, [0, 2]), (9, [1]), (24, [0, 1, 2]),
                                    (8, [0]), (17, [])])
def test_columns_that_ended_cost_no_more_sweeps(tmp_path, p, slow):
    """Packed columns per residual: all, then those of the slow groups only, until these end one after another;
    every column leaves from where it stood."""
    build(PACKED, tmp_path)
    width = lambda q: min(8, p - 8 * q)
    rows, want, left = [], [p], list(slow)
    rows.append([10.0 ** (-6 if c // 8 in slow else -14) for c in range(p)])
    for step in range(2, 2 + len(slow)):
        want.append(sum(width(q) for q in left))
        left = left[1:]
        rows.append([10.0 ** (-6 - 1.5 * step if c // 8 in left else -14) for c in range(p)])
    text = f"{p}\n" + "\n".join(" ".join(map(str, r)) for r in rows) + "\n"
    out = subprocess.run([str(tmp_path / "main")], input=text, capture_output=True, text=True, check=True).stdout
    first, second = out.strip("\n").split("\n")
    assert first.split() == [str(v) for v in want + [0]]
    assert [int(v) for v in second.split()] == list(range(p))
