"""Forces that are infinite, NaN or near the largest double: the populations
are the oracle's, bit for bit where they are finite, infinite and NaN where
its are (the reference multiplies by every component of a direction, and 0
times an infinite force is NaN).

Forces are put into the sheet's records and spread without the force stages,
or come from a sheet whose stretching coefficient overflows."""
import numpy as np
import pytest

import lbib
import pyoracle as P
from pyoracle import Case, centred_sheet

pytestmark = pytest.mark.gpu

NX, NY, NZ = 24, 20, 20
IN = (slice(None), slice(2, NZ - 2), slice(2, NY - 2), slice(2, NX - 2))


def _case(**kw):
    return Case(NX, NY, NZ, [centred_sheet(NX, NY, NZ, 6, 6, 0.9, 9.3)], **kw)


def _moved(s, o):
    rng = np.random.default_rng(2)
    rec = o.sheet().copy()
    rec[..., :3] += rng.uniform(-0.3, 0.3, rec[..., :3].shape)
    return rec


@pytest.mark.parametrize("bulk", ["1", "0"])
@pytest.mark.parametrize("force", [(np.inf, 0.1, 0.2), (0.1, -np.inf, 0.0), (0.0, 0.1, np.inf), (-np.inf, np.inf, 0.1),
                                   (np.nan, 0.1, 0.2), (1e300, 0.1, -1e300), (1e-300, 0.0, 0.1), (1e130, 1e-130, 1.0)])
def test_spread_and_collision(gpu, oracle_built, monkeypatch, bulk, force):
    monkeypatch.setenv("LBIB_FLUID_BULK", bulk)
    case = _case()
    with lbib.Solver(case) as s:
        o = P.Oracle(case, cr_cos=True)
        s.run(3); o.run(3)
        rec = _moved(s, o)
        rec[2, 3, 9:12] = force
        s.set_sheet(0, rec); o.set_sheet(0, rec)
        for n in ["spread", "collide", "stream", "bounceback", "moments", "copy_inout", "replace"]:
            s.stage(n); o.stage(n)
        np.testing.assert_array_equal(s.df1()[IN], o.df(0)[IN])


@pytest.mark.parametrize("overlap", ["2", "3", "0"])
@pytest.mark.parametrize("Ks_l", [1e308, 1e200])
def test_overflowing_stretching(gpu, oracle_built, monkeypatch, overlap, Ks_l):
    monkeypatch.setenv("LBIB_OVERLAP", overlap)
    case = _case(Ks_l=Ks_l, Kb_l=0.0)
    with lbib.Solver(case) as s:
        o = P.Oracle(case, cr_cos=True)
        rec = _moved(s, o)
        s.set_sheet(0, rec); o.set_sheet(0, rec)
        s.run(1)
        o.run(1) if Ks_l < 1e300 else [o.stage(n) for n in (
            "bending", "stretching", "elastic", "spread", "collide", "stream", "bounceback", "copy_inout", "replace")]
        np.testing.assert_array_equal(s.df1()[IN], o.df(0)[IN])
