"""Every launch of a kernel with bounded waits passes a device status word (no GPU: the sources are read).

A stored product or a sweep that gives up writes nothing but that word; without one the call would return
a result that was never computed. The word of a coarse solve is the context's, which its entry points read.
"""
import re

import pytest

from conftest import ROOT

CSRC = ROOT / "treams-rs_b200" / "csrc"


def calls(name):
    """The argument lists of every call of `name` (not its declarations)."""
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"(?<!void )(?<!bool )\b" + name + r"\(", text):
            depth, args, start = 0, [], m.end()
            for i in range(m.end(), len(text)):
                c = text[i]
                if c == "," and depth == 0:
                    args.append(text[start:i].strip())
                    start = i + 1
                elif c in "([{":
                    depth += 1
                elif c in ")]}":
                    if depth == 0:
                        args.append(text[start:i].strip())
                        break
                    depth -= 1
            yield path.name, args


@pytest.mark.parametrize("name,position", [("launch_apply_stored", 13), ("lu_solve_fp64", 9), ("lu_solve_fp32", 9),
                                           ("lu_solve_adjoint_fp64", 9), ("lu_solve_adjoint_fp32", 9)])
def test_calls_pass_a_status_word(name, position):
    found = list(calls(name))
    assert found
    for where, args in found:
        assert len(args) > position and "status" in args[position], (where, args)


def test_coarse_solves_report_where_the_entry_points_read():
    text = (CSRC / "api.cu").read_text()
    body = text[text.index("struct FactorCoarse"):]
    body = body[:body.index("\n};")]
    assert "ctx->d_status" in body and "wk.status" not in body
