"""The term lists' shuffles take whole warps (no GPU): csrc/apply_shapes.h compiled into a small program.

For every shape of the operator's kernels (product form at lmax 2..5, the dipole blocks at lmax 1..10, the
stored product) it lists the threads of a CTA, the tasks and the lanes per task; a warp of which some lanes
have left the loop over tasks must not reach a shuffle over all 32.
"""
import subprocess

import pytest

from conftest import ROOT

CSRC = ROOT / "treams-rs_b200" / "csrc"
PROGRAM = r"""
#include <cstdio>
#include "apply_shapes.h"
using namespace tcu;
static void row(const char* name, int threads, int tile, int tasks, int nsrc) {
    std::printf("%s %d %d %d %d\n", name, threads, tile, tasks, epilogue_lanes(tasks, threads, nsrc));
}
int main() {
    for (int L = 2; L <= 5; ++L) {
        const GemmShape s = gemm_shape(L);
        row("product", shape_threads(s), s.RG * s.CG, s.DI * L * (L + 2), L * (L + 2));
    }
    for (int L = 1; L <= 10; ++L)
        for (int rows = 0; rows < 2; ++rows) {
            const int ndst = rows ? 3 : L * (L + 2), order = 1 + (rows ? 1 : L), ts = (order + 1) * (order + 1);
            const GemmShape s = sub_shape(ts);
            row("dipole", shape_threads(s), s.RG * s.CG, s.DI * ndst, 3);
            if (ts <= 128) row("stored dipole", 288, 256, std::max(1, 128 / ts) * ndst, 3);
        }
    for (int L = 2; L <= 5; ++L) {
        const int ts = (2 * L + 1) * (2 * L + 1), threads = L < 5 ? 288 : 544;
        row("stored", threads, threads - 32, std::max(1, 128 / ts) * L * (L + 2), L * (L + 2));
    }
}
"""


def test_whole_warps_reach_the_shuffles(tmp_path):
    (tmp_path / "main.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", f"-I{CSRC}", str(tmp_path / "main.cpp"), "-o", str(tmp_path / "main")],
                   check=True)
    rows = subprocess.run([str(tmp_path / "main")], capture_output=True, text=True, check=True).stdout.strip()
    assert len(rows.split("\n")) >= 28
    for r in rows.split("\n"):
        threads, tile, tasks, lanes = map(int, r.split()[-4:])
        assert tile <= threads <= 544
        if lanes == 1:
            continue  # no shuffles
        end = (tasks * lanes + 31) // 32 * 32
        for warp in range((threads + 31) // 32):
            passes = {len(range(t, end, threads)) for t in range(32 * warp, min(threads, 32 * warp + 32))}
            assert len(passes) == 1 and (32 * warp + 32 <= threads or passes == {0}), r
