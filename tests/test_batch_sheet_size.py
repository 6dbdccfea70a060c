"""A batch problem's sheet needs four nodes each way: the bending formulas of
nodes 0 and 1 read nodes 2 and 3, which a smaller sheet does not have.  Such
a problem is refused before anything is allocated, as the one-grid solver
refuses it."""
import pytest

import lbib
from pyoracle import Case, Sheet


@pytest.mark.parametrize("rows,cols", [(3, 8), (8, 3), (2, 8), (8, 2), (2, 2), (3, 3)])
def test_small_sheets_are_refused(lbib_built, rows, cols):
    good = Case(32, 16, 16, [Sheet(4, 4, 3.0, 3.0, 10.0, 6.0, 6.0)])
    small = Case(32, 16, 16, [Sheet(rows, cols, 3.0, 3.0, 10.0, 6.0, 6.0)])
    with pytest.raises(lbib.LbibError, match=r"\(-1\)"):
        lbib.Batch([good, small], "f64")
