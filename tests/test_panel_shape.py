"""CTAs of an LU panel on clusters, on the host (no GPU): csrc/panel_shape.h compiled into a small program.

Every shape covers its rows within shared memory, a cluster count that the device holds, and the least rows that the
caller asks for bound the SMs that a panel takes: the workers of a batch ask for 192 so that their panels run side
by side.
"""
import subprocess

import pytest

from conftest import ROOT

CSRC = ROOT / "treams-rs_b200" / "csrc"
PROGRAM = r"""
#include <cstdio>
#include "panel_shape.h"
int main() {
    int entry, rows, nb, least, most;
    while (std::scanf("%d %d %d %d %d", &entry, &rows, &nb, &least, &most) == 5) {
        const tcu::PanelShape s = tcu::panel_cluster_shape(entry, rows, nb, least, most);
        const size_t smem = s.cs ? tcu::panel_cluster_smem(entry, s.chunk, nb, s.cs) : 0;
        std::printf("%d %d %d %d\n", s.cs, s.ncl, s.chunk, (int)(smem <= 224 * 1024));
    }
}
"""
FP32, FP64 = (8, 128), (16, 64)  # bytes of an entry, columns of a panel


@pytest.fixture(scope="module")
def shapes(tmp_path_factory):
    d = tmp_path_factory.mktemp("shape")
    (d / "m.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CSRC}", str(d / "m.cpp"), "-o", str(d / "m")], check=True)

    def ask(asked):
        text = "\n".join(f"{e} {rows} {nb} {least} {most}" for (e, nb), rows, least, most in asked)
        out = subprocess.run([str(d / "m")], input=text, capture_output=True, text=True, check=True).stdout
        return [tuple(map(int, line.split())) for line in out.splitlines()]
    return ask


@pytest.mark.parametrize("kind", [FP32, FP64])
@pytest.mark.parametrize("least", [0, 64, 192, 256])
def test_shapes_cover_their_rows(shapes, kind, least):
    rows = [1, 2, 15, 16, 17, 63, 64, 65, 191, 192, 193, 1023, 1024, 1025, 1920, 3071, 3072, 3073, 4270, 9216, 12576,
            21168]  # 7 clusters of 16 CTAs of 189 rows, the most in FP64
    for r, (cs, ncl, chunk, ok) in zip(rows, shapes([(kind, r, least, 7) for r in rows])):
        assert cs in (1, 2, 4, 8, 16) and 1 <= ncl <= 7 and (ncl == 1 or cs == 16)
        assert chunk <= 256 and ok and cs * ncl * chunk >= r > (cs * ncl - 1) * (chunk - 1)


def test_what_the_device_cannot_hold_is_refused(shapes):
    asked = [(FP32, 22500, 0, 7), (FP64, 22500, 192, 7), (FP32, 4270, 0, 1), (FP32, 100, 0, 0)]
    assert [s[0] for s in shapes(asked)] == [0, 0, 0, 0]


def test_least_rows_bound_the_clusters(shapes):
    asked = [(FP32, 9216, 0, 7), (FP32, 9216, 192, 7), (FP32, 6144, 0, 7), (FP32, 6144, 192, 7), (FP64, 1200, 0, 7),
             (FP64, 1200, 192, 7)]
    assert [s[:2] for s in shapes(asked)] == [(16, 5), (16, 3), (16, 3), (16, 2), (16, 1), (8, 1)]
