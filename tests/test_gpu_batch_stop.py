"""What a batch problem leaves behind when its sheet leaves the grid: the
records of the failing step, forces of every node included, whichever node
failed and whenever its block ran -- the same in every run, and the same as
the problem alone.

The sheets have more chunks of 32 nodes than the chip holds blocks at once
(1250 of at most 4 x 148), or a few; a sheet at the outlet drifts out of its
grid within the steps."""
import numpy as np
import pytest

import lbib
from pyoracle import Case, Sheet, centred_sheet

pytestmark = pytest.mark.gpu


def _bad(rows, cols):
    ny = nz = 64
    w, h = 0.25 * (cols - 1), 0.25 * (rows - 1)
    return Case(32, ny, nz, [Sheet(rows, cols, w, h, 28.6, (ny - 1 - h) / 2, (nz - 1 - w) / 2)], u_l=0.1)


def _batch(cases, steps):
    with lbib.Batch(cases, "f64") as b:
        for n in steps:
            b.run(n)
        codes, step = b.status()
        return [b.sheet(k) for k in range(len(cases))], codes, step


@pytest.mark.parametrize("rows,cols", [(200, 200), (13, 17)])
@pytest.mark.parametrize("steps", [[1, 4, 3, 2, 10], [20]])
def test_records_of_a_stopped_problem(gpu, rows, cols, steps):
    cases = [centred(), _bad(rows, cols), centred()]
    sheets, codes, step = _batch(cases, steps)
    assert list(codes != 0) == [False, True, False] and 1 < step[1] < sum(steps)
    for _ in range(3):
        again, c2, s2 = _batch(cases, steps)
        assert (c2 == codes).all() and (s2 == step).all()
        for a, b in zip(again, sheets):
            np.testing.assert_array_equal(a, b)
    with lbib.Solver(cases[1]) as s:
        with pytest.raises(lbib.LbibError):
            s.run(sum(steps))
        np.testing.assert_array_equal(sheets[1], s.sheet())


def centred():
    return Case(32, 16, 16, [centred_sheet(32, 16, 16, 8, 8, 0.5, 10.0)])
