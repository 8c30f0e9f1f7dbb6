"""The stored product's block lists and what its warps hold, on the host (no GPU): the library's own list
builder, called from a small C++ program that links it.

A list longer than warps x slots would lose its last blocks silently. Every lmax of the full operator fits;
a plan whose terms read every table entry of every source does not, except at lmax 2, whose warps hold the
whole product, and is refused.
"""
import subprocess

import pytest

from conftest import ROOT

CSRC = ROOT / "treams-rs_b200" / "csrc"
PROGRAM = r"""
#include <cstdio>
#include "plan.h"
namespace tcu { bool stored_product_blocks(const DevPlan& P, const HostPlan& h, ProductBlocks* b); }
int main() {
    for (int L = 2; L <= 7; ++L)
        for (int all = 0; all < 2; ++all) {
            tcu::HostPlan h = tcu::build_plan(L);
            tcu::DevPlan d{};
            d.L = L, d.nlm = h.nlm, d.order = h.order, d.tsize = (h.order + 1) * (h.order + 1);
            if (all) {  // every (source, destination 0) reads every entry
                h.idx.clear();
                for (size_t c = 0; c < h.combo.size() / 2; ++c) {
                    const bool reads = c % h.nlm == 0;
                    h.combo[2 * c] = (int)h.idx.size();
                    h.combo[2 * c + 1] = reads ? d.tsize : 0;
                    for (int t = 0; reads && t < d.tsize; ++t) h.idx.push_back((uint16_t)t);
                }
            }
            static tcu::ProductBlocks b;
            const bool ok = tcu::stored_product_blocks(d, h, &b);
            std::printf("%d %d %d %d %d\n", L, all, (int)ok, b.count[0], b.count[1]);
        }
}
"""
HOLDS = {2: 8 * 4, 3: 8 * 6, 4: 8 * 7, 5: 16 * 7, 6: 16 * 7, 7: 16 * 7}
ALL = {2: 13 * 2, 3: 13 * 4, 4: 11 * 6, 5: 16 * 9, 6: 22 * 6, 7: 29 * 4}


@pytest.fixture(scope="module")
def lists(tmp_path_factory):
    import treams_b200
    d = tmp_path_factory.mktemp("blocks")
    lib = treams_b200.library_path()
    (d / "main.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", f"-I{CSRC}", "-I/usr/local/cuda/include", str(d / "main.cpp"), str(lib),
                    f"-Wl,-rpath,{lib.parent}", "-o", str(d / "main")], check=True)
    out = subprocess.run([str(d / "main")], capture_output=True, text=True, check=True).stdout
    return {tuple(map(int, row.split()[:2])): tuple(map(int, row.split()[2:])) for row in out.strip().split("\n")}


@pytest.mark.parametrize("lmax", range(2, 8))
def test_the_plans_lists_fit(lists, lmax):
    ok, first, second = lists[lmax, 0]
    assert ok and 0 < first <= HOLDS[lmax] and 0 <= second <= HOLDS[lmax] and (second > 0) == (lmax == 7)


@pytest.mark.parametrize("lmax", range(2, 8))
def test_a_list_that_does_not_fit_is_refused(lists, lmax):
    ok, first, second = lists[lmax, 1]
    assert bool(ok) == (ALL[lmax] <= HOLDS[lmax])
    assert max(first, second) <= HOLDS[lmax]
