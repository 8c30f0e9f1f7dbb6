"""Row interchanges after a panel that gave up: pivots that no panel can have chosen move nothing.

The self-test runs the interchange kernel on 96 rows with pivots of -1, n, the largest and smallest
32-bit numbers and rows above the column, and one valid interchange among them, between guards; it
reports a wrongly moved entry as an error other than the wait's own. Exact: the entries are whole numbers.
"""
import pytest

pytestmark = pytest.mark.gpu


def test_interchanges_without_valid_pivots_move_nothing(ctx):
    import treams_b200 as t
    with pytest.raises(t.TreamsCudaError, match="gave up"):
        ctx.wait_selftest(0.01)
