"""The one-launch ghost fill against the reference's order of fills (periodic
halos along i, j, k, then face by face, src/boundary_exchange.c and
src/boundary_conditions.c), restated here with numpy: every point of every
field, edges and corners included, exactly (the fill copies, negates and sets
constants).  Grids of the smallest and of odd sizes, all kinds mixed, gas and
face field with kinds of their own, the entropy channel live."""
import math

import numpy as np
import pytest

from conftest import NG

pytestmark = pytest.mark.gpu


def _fill(n, W, B, gas, gem):
    """In place; gas and gem are six kinds each."""
    fields = [(W[m], -1, gas, m) for m in range(6)] + [(B[c], c, gem, c) for c in range(3)]

    def at(t, a, i):
        s = [slice(None)] * 3
        s[a] = i
        return t[tuple(s)]

    for a in range(3):
        if gas[2 * a] != "p":
            continue
        for t, fa, _, _ in fields:
            o = int(fa == a)
            for l in range(NG):
                at(t, a, n[a] + NG + o + l)[:] = at(t, a, NG + o + l)
                at(t, a, l)[:] = at(t, a, n[a] + l)
    for face in range(6):
        a, up = face // 2, face % 2
        if gas[2 * a] == "p":
            continue
        for t, fa, kinds, m in fields:
            k, o, cell = kinds[face], int(fa == a), fa < 0
            if k == "n" or (k == "r" and not cell) or (k == "f" and cell and m == 5):
                continue
            for l in range(NG):
                dst = n[a] + NG + l + o if up else l
                if k == "f":
                    v = 0.0
                    if cell and m == 0:
                        v = 2.0 if (a, up) == (1, 0) else 1.0
                    elif cell and m == 4:
                        v = 2.5 if (a, up) == (1, 1) else 1.0
                    at(t, a, dst)[:] = v
                    continue
                if k == "e":
                    v = at(t, a, n[a] + NG - 1 + o if up else NG).copy()
                else:
                    v = at(t, a, n[a] + NG - 1 - l if up else 2 * NG - 1 - l + o).copy()
                if k == "o":  # half a turn in phi, theta and phi components turned
                    v = v[:, NG + (np.arange(v.shape[1]) - NG + n[2] // 2) % n[2]]
                    if m in (2, 3) if cell else m != 0:
                        v = -v
                if k == "r" and cell and m == 1 + a:
                    v = -v
                at(t, a, dst)[:] = v


CASES = [("pppppp", ""), ("eeeeee", ""), ("srfepp", ""), ("ppsrne", ""), ("ffrree", "ssnnff"), ("rrffss", "eerrnn"),
         ("nnnnnn", ""), ("fepprs", "ffppen"), ("enrfsf", "rsefnr")]


@pytest.mark.parametrize("n", [(4, 4, 4), (5, 9, 4), (33, 6, 17)])
@pytest.mark.parametrize("bc,gem", CASES)
def test_fill_in_one_launch_equals_the_fills_in_turn(n, bc, gem):
    import gop

    rng = np.random.default_rng(sum(n) + len(bc + gem) + ord(bc[0]) + ord(bc[5]))
    N = tuple(m + 2 * NG + 1 for m in n)
    W, B = rng.uniform(0.5, 1.5, (6,) + N), rng.uniform(-0.1, 0.1, (3,) + N)
    xs = [gop.grid_uniform(m, 0.0, 1.0) for m in n]
    inst = gop.Instance(n, *xs, bc=bc, gem_bc=gem)
    inst.upload(W, B)
    inst.prepare()
    d = inst.download(("gas", "face_b"))
    inst.close()
    _fill(n, W, B, bc, gem or bc)
    np.testing.assert_array_equal(d["gas"], W)
    np.testing.assert_array_equal(d["face_b"], B)


def test_pole_fill():
    import gop

    n = (8, 16, 32)
    rng = np.random.default_rng(5)
    N = tuple(m + 2 * NG + 1 for m in n)
    W, B = rng.uniform(0.5, 1.5, (6,) + N), rng.uniform(-0.1, 0.1, (3,) + N)
    W[5] = 0.0
    xs = [gop.grid_uniform(n[0], 1.0, 2.0), gop.grid_uniform(n[1], 0.0, math.pi),
          gop.grid_uniform(n[2], 0.0, 2.0 * math.pi)]
    inst = gop.Instance(n, *xs, coord=gop.COORD_SPHERICAL, bc="eeoopp", ring_average=True)
    inst.upload(W, B)
    inst.prepare()
    d = inst.download(("gas", "face_b"))
    inst.close()
    _fill(n, W, B, "eeoopp", "eeoopp")
    np.testing.assert_array_equal(d["gas"], W)
    np.testing.assert_array_equal(d["face_b"], B)


@pytest.mark.parametrize("bc", ["pppppp", "nnnnnn", "eesspp"])
def test_steps_end_and_begin_with_the_fill(bc):
    """Steps one by one, in one call, with a stop time, and none at all: the
    same state, time and step count."""
    import gop

    n = (12, 8, 6)
    rng = np.random.default_rng(7)
    N = tuple(m + 2 * NG + 1 for m in n)
    W, B = np.ones((6,) + N), np.full((3,) + N, 0.3)
    W[5] = 0.0
    W[1:4] = 0.1 * rng.standard_normal((3,) + N)
    xs = [gop.grid_uniform(m, 0.0, 1.0) for m in n]
    out = []
    for way in range(4):
        inst = gop.Instance(n, *xs, bc=bc)
        inst.upload(W, B)
        inst.prepare()
        if way == 0:
            t = inst.step(5)
        elif way == 1:
            for _ in range(5):
                inst.step(0)
                t = inst.step(1)
        elif way == 2:
            t4 = inst.step(4)
            t = inst.step(10, time_stop=t4)  # the step that takes time past t4 is the last
        else:
            inst.step(2)
            inst.autotune(reps=1)
            t = inst.step(3)
        st = inst.stats()
        assert st["steps"] == 5 and st["time"] == t
        out.append((inst.download(("gas", "face_b", "gas_p")), t, st["dt"], st["divb_max"]))
        inst.close()
    for d, t, dt, divb in out[1:]:
        assert (t, dt) == out[0][1:3]
        for f in ("gas", "face_b", "gas_p"):
            np.testing.assert_allclose(d[f], out[0][0][f], rtol=0, atol=1e-13)
