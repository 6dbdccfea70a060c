"""Tiles that more nodes touch than the gather's lists hold at once (256 chunks
of 32 nodes, 1024 nodes): a list at a time, bit for bit against the oracle
with the correctly rounded cosine, and in a time that does not depend on how
the nodes came to lie together -- visited one chunk after another, the sheet
of the last test took 115 times a flat one's step."""
import time

import numpy as np
import pytest

import lbib
import pyoracle as P

pytestmark = pytest.mark.gpu

NX, NY, NZ = 32, 40, 44


def _case(rows, cols):
    return P.Case(NX, NY, NZ, [P.Sheet(rows, cols, 30.0, 26.0, 12.0, 6.5, 6.5)], Ks_l=1e-6, Kb_l=1e-7)


def _strewn(rows, cols, lo, hi):
    return np.random.default_rng(rows + cols).uniform(lo, hi, (rows, cols, 3))


# nodes, chunks and where: all in one stencil start (every node on the same tiles), or over a few
@pytest.mark.parametrize("rows,cols", [
    (32, 32),     # 1024 nodes: the list exactly full
    (25, 41),     # 1025: one more, the last in a chunk of its own
    (64, 128),    # 8192 nodes, 256 chunks: the chunks exactly full
    (64, 129),    # 258 chunks
    (41, 313),    # 12833 nodes, 402 chunks, the last of one node
])
@pytest.mark.parametrize("hi", [(14.9, 20.9, 20.9), (19.0, 25.0, 25.0)])
def test_full_lists(gpu, oracle_built, rows, cols, hi):
    case = _case(rows, cols)
    pos = _strewn(rows, cols, (14.1, 20.1, 20.1), hi)
    o = P.Oracle(case, cr_cos=True)
    with lbib.Solver(case) as s:
        rec = s.sheet()
        rec[..., :3] = pos
        s.set_sheet(0, rec)
        o.set_sheet(0, rec)
        for n in ["bending", "stretching", "elastic", "spread"]:
            s.stage(n)
            o.stage(n)
        for a, b in zip(s.force(), o.force()):
            np.testing.assert_array_equal(a, b)


def test_full_lists_in_a_batch(gpu):
    """The second problem's chunks start inside the batch's."""
    big = P.Case(NX, NY, NZ, [P.Sheet(64, 129, 0.9, 0.9, 14.0, 20.05, 20.05)], Ks_l=1e-9, Kb_l=1e-12)
    other = P.Case(32, 16, 16, [P.centred_sheet(32, 16, 16, 8, 8, 0.5, 10.0)])
    with lbib.Batch([other, big, other], "f64") as b, lbib.Solver(big) as s:
        b.run(3)
        s.run(3)
        for x, y in zip(b.moments(1) + [b.sheet(1)], s.moments() + [s.sheet()]):
            np.testing.assert_array_equal(x, y)


def test_time_of_strewn_nodes(gpu):
    nx, ny, nz = 128, 96, 96
    took = []
    for strewn in (False, True):
        case = P.Case(nx, ny, nz, [P.centred_sheet(nx, ny, nz, 104, 104, 0.5, 40.0)], u_l=1e-5, Ks_l=1e-12, Kb_l=1e-12)
        with lbib.Solver(case) as s:
            if strewn:
                rec = s.sheet()
                rec[..., :3] = _strewn(104, 104, (2.0, 2.0, 2.0), (nx - 4.0, ny - 4.0, nz - 4.0))
                s.set_sheet(0, rec)
            s.run(4)
            s.synchronize()
            best = 1e9
            for _ in range(5):
                t = time.perf_counter()
                s.run(4)
                s.synchronize()
                best = min(best, time.perf_counter() - t)
            took.append(best)
    assert took[1] < 40 * took[0]     # about 10 times; 115 before
