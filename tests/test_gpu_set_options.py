"""Options and parameters changed between steps: the next step's box, which
the last move left, was made for the options before (a ring of tiles around
it only where the streams join after the move, never with periodic z).

The step that joins its streams late against the stages in order, bit for
bit, with the periodic-z option dropped and the elasticity changed midway."""
import numpy as np
import pytest

import lbib
import pyoracle as P
from pyoracle import Case, Sheet

pytestmark = pytest.mark.gpu
PERIODIC = 0x100


def _run(monkeypatch, overlap, start, then, dims):
    monkeypatch.setenv("LBIB_OVERLAP", overlap)
    nx, ny, nz = dims
    case = Case(nx, ny, nz, [Sheet(18, 20, 9.5, 8.5, 14.0, 12.0, 14.0)], Ks_l=0.02, Kb_l=0.002, compat=start)
    s = lbib.Solver(case)
    s.run(5)
    assert s.lib.lbib_set_compat(s.gv, then) == 0
    s.run(5)
    assert s.lib.lbib_set_params(s.gv, 0.6, 0.01, 0.05, 0.001) == 0
    s.run(5)
    out = s.moments() + [s.sheet()]
    s.close()
    return out


@pytest.mark.parametrize("dims", [(48, 40, 44), (128, 64, 64)])
@pytest.mark.parametrize("start,then", [(P.COMPAT_ALL | PERIODIC, P.COMPAT_ALL), (P.COMPAT_ALL, 0)])
def test_late_join_after_a_change(gpu, monkeypatch, start, then, dims):
    late = _run(monkeypatch, "3", start, then, dims)
    plain = _run(monkeypatch, "0", start, then, dims)
    for a, b in zip(late, plain):
        np.testing.assert_array_equal(a, b)


def test_box_is_made_anew(gpu, monkeypatch):
    """The step after the change has the launch that computes the box."""
    case = Case(48, 40, 44, [Sheet(18, 20, 9.5, 8.5, 14.0, 12.0, 14.0)])
    monkeypatch.setenv("LBIB_OVERLAP", "2")
    with lbib.Solver(case) as s:
        s.run(3)
        n = s.kernel_launches
        s.run(1)
        plain = s.kernel_launches - n
        assert s.lib.lbib_set_compat(s.gv, 0) == 0
        n = s.kernel_launches
        s.run(1)
        assert s.kernel_launches - n == plain + 1
