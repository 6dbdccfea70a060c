"""Hosts that drive the step by its stages, leave some out or repeat them.

A spread fills one of two buffers (tile map, tile list); what the stages
after it do or leave undone must not reach the next spread into the same
buffer: its list holds the tiles that its own nodes touch, each once, and
forces and fields are the oracle's, bit for bit."""
import numpy as np
import pytest

import lbib
import pyoracle as P
from pyoracle import Case, Sheet

pytestmark = pytest.mark.gpu

NX, NY, NZ = 40, 24, 28           # 420 tiles; 16 nodes: a list holds 8 * 16
FLUID = ["collide", "stream", "bounceback", "moments", "copy_inout", "replace"]


def _case():
    return Case(NX, NY, NZ, [Sheet(4, 4, 6.0, 6.0, 12.0, 8.0, 9.0)])


def _list_length(s, tmp_path):
    """The tile list's length, from the restart file: magic, 8 ints, 8
    doubles, the sheet's shape, then 6 ints of which it is the last."""
    path = str(tmp_path / "state.rst")
    s.save(path)
    with open(path, "rb") as f:
        f.seek(8 + 8 * 4 + 8 * 8 + 2 * 4)
        return int(np.frombuffer(f.read(24), np.int32)[5])


def _touched(pos):
    """Tiles of 4^3 cells that the stencils of nodes at pos touch."""
    lo = np.floor(pos.reshape(-1, 3) - 2).astype(int) + 1
    t = set()
    for a in lo:
        r = [range(v >> 2, ((v + 3) >> 2) + 1) for v in a]
        t |= {(x, y, z) for x in r[0] for y in r[1] for z in r[2]}
    return len(t)


def _place(s, o, rng):
    """The sheet somewhere else, bent."""
    rec = o.sheet().copy()
    at = rec[..., :3] - rec[..., :3].mean(axis=(0, 1))
    mid = rng.uniform([7.0, 8.0, 8.0], [NX - 8.0, NY - 9.0, NZ - 9.0])
    rec[..., :3] = at + mid + rng.uniform(-0.05, 0.05, at.shape)
    s.set_sheet(0, rec)
    o.set_sheet(0, rec)
    return rec[..., :3]


def _both(s, o, names):
    for n in names:
        s.stage(n)
        o.stage(n)


def _same(s, o):
    for a, b in zip(s.force() + s.moments(), o.force() + o.moments()):
        np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(s.sheet(), o.sheet())


@pytest.mark.parametrize("again", [[], ["moments"], ["moments", "move"]])
@pytest.mark.parametrize("overlap", ["2", "3", "0"])
def test_steps_with_a_placed_sheet(gpu, oracle_built, tmp_path, monkeypatch, overlap, again):
    """No move (the host places the sheet), or moments and a move more than
    a step has; full steps before, between and after."""
    monkeypatch.setenv("LBIB_OVERLAP", overlap)
    rng = np.random.default_rng(5)
    with lbib.Solver(_case()) as s:
        o = P.Oracle(_case(), cr_cos=True)
        s.run(3); o.run(3)
        for t in range(40):
            pos = _place(s, o, rng)
            _both(s, o, ["bending", "stretching", "elastic", "spread"])
            assert _list_length(s, tmp_path) == _touched(pos)
            _both(s, o, FLUID)
            if t % 4 == 0:
                for n in again:          # the oracle's moments belong between bounceback and replace
                    s.stage(n)
                if "move" in again:
                    o.stage("move")
            _same(s, o)
            if t % 7 == 6:
                s.run(2); o.run(2)
                _same(s, o)


def test_moments_before_the_collision(gpu, oracle_built):
    """Moments asked for between a spread and its collision leave the old
    map to the collision."""
    rng = np.random.default_rng(6)
    with lbib.Solver(_case()) as s:
        o = P.Oracle(_case(), cr_cos=True)
        s.run(3); o.run(3)
        for _ in range(4):
            _place(s, o, rng)
            _both(s, o, ["bending", "stretching", "elastic", "spread"])
            s.stage("moments")
            _both(s, o, FLUID)
            _same(s, o)


def test_spreads_alone(gpu, oracle_built, tmp_path):
    """Forces asked for at one placement after another, no fluid step."""
    rng = np.random.default_rng(7)
    with lbib.Solver(_case()) as s:
        o = P.Oracle(_case(), cr_cos=True)
        s.run(3); o.run(3)
        for _ in range(40):
            pos = _place(s, o, rng)
            _both(s, o, ["bending", "stretching", "elastic", "spread"])
            assert _list_length(s, tmp_path) == _touched(pos)
            for a, b in zip(s.force(), o.force()):
                np.testing.assert_array_equal(a, b)
