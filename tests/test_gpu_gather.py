"""The spread's node lists where they change form, bit for bit against the
oracle with the correctly rounded cosine: sheets of more than 128 chunks of
32 nodes (boxes of 1024 nodes are tested first), nodes scattered over the
grid (every chunk's box meets every tile: more than the 64 chunks whose
stencil starts are kept, and more than the 256 the list holds, which takes
the scan), more than 1024 nodes on one tile (the scan too), exactly one
chunk, and more pinned sheets than one move launch takes (4)."""
import numpy as np
import pytest

import lbib
import pyoracle as P

pytestmark = pytest.mark.gpu

NX, NY, NZ = 32, 40, 44


def _sheet(rows, cols, x0, w=30.0, h=26.0):
    return P.Sheet(rows, cols, w, h, x0, (NY - 1 - h) / 2, (NZ - 1 - w) / 2)


def _run(case, positions, steps=3):
    s = lbib.Solver(case)
    o = P.Oracle(case, cr_cos=True)
    for k, pos in enumerate(positions):
        if pos is None:
            continue
        rec = s.sheet(k)
        rec[..., :3] = pos
        s.set_sheet(k, rec)
        o.set_sheet(k, rec)
    s.run(steps)
    o.run(steps)
    for a, b in zip(s.moments(), o.moments()):
        np.testing.assert_array_equal(a, b)
    for k in range(len(case.sheets)):
        np.testing.assert_array_equal(s.sheet(k), o.sheet(k))
    s.close()


@pytest.mark.parametrize("rows,cols,lo,hi", [
    (4, 8, None, None),                                       # one chunk
    (72, 72, None, None),                                     # 162 chunks, a flat sheet
    (40, 60, (3, 4, 4), (NX - 5, NY - 5, NZ - 5)),            # 75 chunks, each over the whole grid
    (100, 100, (3, 4, 4), (NX - 5, NY - 5, NZ - 5)),          # 313 chunks, each over the whole grid
    (50, 50, (14.2, 20.1, 20.3), (17.7, 23.6, 23.9)),         # 2500 nodes on a few tiles
])
def test_node_lists(gpu, oracle_built, rows, cols, lo, hi):
    pos = None
    if lo is not None:
        rng = np.random.default_rng(rows)
        pos = rng.uniform(lo, hi, (rows, cols, 3))
    case = P.Case(NX, NY, NZ, [_sheet(rows, cols, 12.0)], Ks_l=1e-6, Kb_l=1e-7)
    _run(case, [pos])


def test_five_pinned_sheets(gpu, oracle_built):
    sheets = [_sheet(9 + k, 11, 5.0 + 4 * k, 8.0, 6.0) for k in range(5)]
    case = P.Case(NX, NY, NZ, sheets, Ks_l=0.01, Kb_l=0.001, compat=P.COMPAT_ALL | 0x400)
    _run(case, [None] * 5, steps=5)


@pytest.mark.parametrize("ks", [1e-150, 1e-305])
def test_tiny_forces(gpu, oracle_built, ks):
    """Forces too small for the divisions by a multiplication with the
    reciprocal (residuals would underflow) take true divisions."""
    rng = np.random.default_rng(3)
    case = P.Case(NX, NY, NZ, [_sheet(12, 14, 12.0)], Ks_l=ks, Kb_l=ks / 10)
    y, z = np.meshgrid(np.linspace(8, 30, 12), np.linspace(8, 34, 14), indexing="ij")
    pos = np.stack([np.full_like(y, 12.0), y, z], axis=-1) + rng.uniform(-0.3, 0.3, y.shape + (3,))
    _run(case, [pos])


@pytest.mark.parametrize("nx,ny,nz,where", [
    (32, 40, 44, (3.0, 6.0, 8.0)),           # at the inlet
    (32, 40, 44, (NX - 4.0, 6.0, 8.0)),      # at the outlet
    (32, 40, 44, (14.0, 3.0, 4.0)),          # in a corner of the walls
    (36, 40, 44, (17.5, 16.0, 15.0)),
    (128, 64, 64, (40.0, 20.0, 18.0)),       # large enough to join late by itself
])
@pytest.mark.parametrize("options", [0, 0x100, 0x400])
def test_streams_joined_after_the_move(gpu, monkeypatch, nx, ny, nz, where, options):
    """The step whose streams join after the move against the stages in order,
    bit for bit, with a sheet that jumps from one end of the grid to another
    (the map of the step before lies outside the box) and back."""
    def run(mode):
        monkeypatch.setenv("LBIB_OVERLAP", mode)
        case = P.Case(nx, ny, nz, [P.Sheet(18, 20, 17.0, 14.0, *where)], Ks_l=0.01, Kb_l=0.001,
                      compat=P.COMPAT_ALL | options)
        s = lbib.Solver(case)
        s.run(4)
        rec = s.sheet(0)
        rec[..., 0] = (nx - 1) - rec[..., 0]
        s.set_sheet(0, rec)
        s.run(3)
        rec = s.sheet(0)
        rec[..., 0] = (nx - 1) - rec[..., 0]
        s.set_sheet(0, rec)
        s.run(4)
        out = [*s.moments(), s.sheet(0)]
        s.close()
        return out
    for a, b in zip(run("3"), run("0")):
        np.testing.assert_array_equal(a, b)
