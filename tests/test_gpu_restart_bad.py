"""Restart files that end early or hold an index out of range are refused,
and the state they were loaded into stays usable: later spreads give the
oracle's forces, a good file continues bit for bit.

The offsets follow the layout in csrc/lbib_device.cu: magic, 8 ints, 8
doubles, a sheet's shape, 6 ints, a long, the populations, the two tables,
the map, the list."""
import struct

import numpy as np
import pytest

import lbib
import pyoracle as P
from cases import small_case

pytestmark = pytest.mark.gpu

NX, NY, NZ = 32, 16, 16
MAP = 8 + 32 + 64 + 8 + 24 + 8 + 8 * 19 * NX * NY * NZ + 2 * 8 * 19 * NY * NZ
TILES = NX // 4 * (NY // 4) * (NZ // 4)
LIST = MAP + 4 * TILES


def _spread_is_right(s, o):
    rng = np.random.default_rng(1)
    for _ in range(3):                   # each buffer at least once
        rec = o.sheet().copy()
        rec[..., :3] += rng.uniform(-0.5, 0.5, 3)
        s.set_sheet(0, rec)
        o.set_sheet(0, rec)
        for n in ["bending", "stretching", "elastic", "spread"]:
            s.stage(n)
            o.stage(n)
        for a, b in zip(s.force(), o.force()):
            np.testing.assert_array_equal(a, b)


def _damage(data, how):
    if isinstance(how, int):
        return data[:how]
    at, value = how
    return data[:at] + struct.pack("<i", value) + data[at + 4:]


@pytest.mark.parametrize("how", [LIST - 4 * TILES // 3, LIST + 8, (LIST + 4, TILES), (LIST, -1), (MAP + 40, -2),
                                 (MAP + 4 * TILES - 4, TILES), 200])
@pytest.mark.parametrize("steps", [6, 7])
def test_bad_file_is_refused(gpu, oracle_built, tmp_path, how, steps):
    good, bad = tmp_path / "good.rst", tmp_path / "bad.rst"
    case = small_case(NX, NY, NZ, 8, 8, 10.0)
    with lbib.Solver(case) as s:
        s.run(steps)
        s.save(str(good))
        s.run(4)
        want = s.moments() + [s.sheet()]
    data = good.read_bytes()
    bad.write_bytes(_damage(data, how))
    o = P.Oracle(case, cr_cos=True)
    with lbib.Solver(case) as s:
        s.run(5)
        with pytest.raises(lbib.LbibError):
            s.load(str(bad))
        _spread_is_right(s, o)
        s.load(str(good))
        s.run(4)
        for a, b in zip(s.moments() + [s.sheet()], want):
            np.testing.assert_array_equal(a, b)
